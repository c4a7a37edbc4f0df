// FP32 sweeps of one-sided block Jacobi through the blocks' Gram matrices (the
// first phase of the refined SVD of large real problems).
//
// Rotating column pairs one by one costs a dot product over the whole column, a
// warp reduction and a barrier per round (1,900 to 2,800 cycles at 301 to 512
// columns), and moves every column of V along.  Here a block step
//   1. forms the Gram matrix of its 2 b columns (2 b <= 32) once,
//   2. runs the step's rounds of rotations on that matrix alone: one thread per
//      pair derives (c, s), then one thread per 2 x 2 block updates it (two CTA
//      barriers, ~400 cycles a round, whatever the column length), while the
//      other threads accumulate the 2 b x 2 b rotation product J,
//   3. multiplies the columns by J, storing them straight where the next step
//      needs them, and writes J to memory.
// V = product of all J is formed afterwards by a kernel whose CTAs own rows of V:
// a row passes through every step's J without any exchange.
// The dot products are those of the columns themselves at every step, so small
// columns keep their relative accuracy; within a step the two-sided updates keep
// it to FP32 of sqrt(g_ii g_jj), well inside the pair tolerance.  The pair order
// (cross pairs of the two blocks at each step, pairs inside the blocks at a
// sweep's first) is that of the column-by-column kernels.
//
//  cluster form: 16 CTAs, two blocks of b columns each (up to 512 columns);
//    step 3 stores into the next owners' shared memory (two buffers, one cluster
//    barrier a step).
//  grid form: one CTA per pair of 8-column blocks, through L2, with a release
//    flag per block (larger problems).
#include <cooperative_groups.h>

#include <algorithm>

#include "plom_common.cuh"
#include "plom_df.cuh"
#include "plom_jacobi.cuh"

namespace cg = cooperative_groups;

namespace plom {

constexpr int JG_THREADS = 512;
constexpr int JG_MAX_SWEEPS = 16;
constexpr int JG_CLUSTER = 16;
constexpr uint64_t JG_WAIT_NS = 2000000000ull;

struct JgArgs {
  const double* A;  // n x n: its rows are the columns to rotate
  int n, b, nblk, pitch;
  float tol, floor, tstop;
  int max_sweeps;
  float* J;       // [sweep][step][pair][2b][2b]: J transposed (row = new column)
  int* nsteps;    // block steps taken
  unsigned long long* amax;
  int* info;
  // grid form
  float* At;      // nblk b x pitch
  int* bflag;
  int* abortf;
  int* counts;    // [JG_MAX_SWEEPS]
  unsigned *cmax, *tmax;
};

// Gram matrix of TB columns of `len` (a multiple of 128) values: warps take 4 x 4
// blocks of it, lanes 16-byte vectors of the columns
template <int TB>
__device__ __forceinline__ void jg_gram(const float* X, int pitch, float (*G)[TB + 1]) {
  constexpr int NB = TB / 4, NT = NB * (NB + 1) / 2;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  for (int t = warp; t < NT; t += JG_THREADS / 32) {
    int bi = 0, r = t;
    while (r >= NB - bi) {
      r -= NB - bi;
      ++bi;
    }
    const int bj = bi + r;
    float acc[16];
#pragma unroll
    for (int q = 0; q < 16; ++q) acc[q] = 0.f;
    for (int v = lane; v < pitch / 4; v += 32) {
      float4 x[4], y[4];
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        x[q] = reinterpret_cast<const float4*>(X + (size_t)(4 * bi + q) * pitch)[v];
        y[q] = reinterpret_cast<const float4*>(X + (size_t)(4 * bj + q) * pitch)[v];
      }
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j)
          acc[4 * i + j] = fmaf(x[i].x, y[j].x, fmaf(x[i].y, y[j].y, fmaf(x[i].z, y[j].z, fmaf(x[i].w, y[j].w, acc[4 * i + j]))));
    }
    // sum 16 values over the warp: halve the values held at each of 4 steps,
    // then add the two half-warps
#pragma unroll
    for (int s = 0; s < 4; ++s) {
      const int o = 16 >> s, h = 8 >> s;  // lane distance, values kept
      const bool up = (lane & o) != 0;
#pragma unroll
      for (int q = 0; q < 8; ++q) {
        if (q >= h) continue;
        const float send = up ? acc[q] : acc[q + h];
        const float keep = up ? acc[q + h] : acc[q];
        acc[q] = keep + __shfl_xor_sync(0xffffffffu, send, o);
      }
    }
    const float g = acc[0] + __shfl_xor_sync(0xffffffffu, acc[0], 1);
    if ((lane & 1) == 0) {
      // lane bits 4, 3, 2, 1 select value bits 3, 2, 1, 0
      const int q = (((lane >> 4) & 1) << 3) | (((lane >> 3) & 1) << 2) | (((lane >> 2) & 1) << 1) | ((lane >> 1) & 1);
      const int i = 4 * bi + (q >> 2), j = 4 * bj + (q & 3);
      G[i][j] = g;
      G[j][i] = g;
    }
  }
}

// the rounds of one block step on G (TB x TB), accumulating Jt (row = new
// column); returns in thread k < b its rotations and largest |t| above the floor
template <int TB>
__device__ __forceinline__ void jg_rounds(float (*G)[TB + 1], float (*Jt)[TB], float2* cs, int2* pq,
                                          bool first, float tol, float floor2, int& rot,
                                          float& tmax) {
  constexpr int B = TB / 2;
  const int tid = threadIdx.x;
  for (int e = tid; e < TB * TB; e += JG_THREADS) Jt[e / TB][e % TB] = (e / TB == e % TB) ? 1.f : 0.f;
  const int nintra = first ? B - 1 : 0;
  for (int rd = 0; rd < nintra + B; ++rd) {
    if (tid < B) {
      int p, q;
      if (rd < nintra) {
        const int h = tid >= B / 2 ? B : 0;
        rr_pair(rd, tid % (B / 2), B, p, q);
        p += h;
        q += h;
      } else {
        p = tid;
        q = tid + rd - nintra;
        q = B + (q >= B ? q - B : q);
      }
      const float al = G[p][p], be = G[q][q], g = G[p][q];
      float c = 1.f, s = 0.f, t = 0.f;
      if (al > 0.f && be > 0.f && fabsf(g) > tol * (al * rsqrtf(al)) * (be * rsqrtf(be))) {
        const float z = __fdividef(be - al, 2.0f * g);
        const float az = fabsf(z), w = fmaf(z, z, 1.0f);
        t = az > 1e18f ? __fdividef(0.5f, z) : copysignf(__fdividef(1.0f, az + w * rsqrtf(w)), z);
        const float w1 = fmaf(t, t, 1.0f), c0 = rsqrtf(w1);
        c = fmaf(0.5f * c0, fmaf(-w1 * c0, c0, 1.0f), c0);
        s = c * t;
        ++rot;
        if (fmaxf(al, be) > floor2) tmax = fmaxf(tmax, fabsf(t));
      }
      cs[tid] = make_float2(c, s);
      pq[tid] = make_int2(p, q);
    }
    __syncthreads();
    if (tid < 256) {
      if (tid < B * B) {
        const int k = tid / B, l = tid % B;
        const float2 rk = cs[k], rl = cs[l];
        const int2 a = pq[k], c = pq[l];
        const float g00 = G[a.x][c.x], g01 = G[a.x][c.y], g10 = G[a.y][c.x], g11 = G[a.y][c.y];
        // columns, then rows: x' = c x - s y, y' = s x + c y
        const float h00 = fmaf(rl.x, g00, -rl.y * g01), h01 = fmaf(rl.y, g00, rl.x * g01);
        const float h10 = fmaf(rl.x, g10, -rl.y * g11), h11 = fmaf(rl.y, g10, rl.x * g11);
        float f00 = fmaf(rk.x, h00, -rk.y * h10), f10 = fmaf(rk.y, h00, rk.x * h10);
        float f01 = fmaf(rk.x, h01, -rk.y * h11), f11 = fmaf(rk.y, h01, rk.x * h11);
        if (k == l && rk.y != 0.f) f01 = f10 = 0.f;
        G[a.x][c.x] = f00;
        G[a.x][c.y] = f01;
        G[a.y][c.x] = f10;
        G[a.y][c.y] = f11;
      }
    } else {
      for (int e = tid - 256; e < TB * B; e += 256) {
        const int l = e / TB, i = e % TB;
        const float2 r = cs[l];
        const int2 c = pq[l];
        const float x = Jt[c.x][i], y = Jt[c.y][i];
        Jt[c.x][i] = fmaf(r.x, x, -r.y * y);
        Jt[c.y][i] = fmaf(r.y, x, r.x * y);
      }
    }
    __syncthreads();
  }
}

// X J for the rows of X (TB columns of `len` values): put(j, r, value)
template <int TB, typename Put>
__device__ __forceinline__ void jg_apply(const float* X, int pitch, int len, const float (*Jt)[TB],
                                         Put&& put) {
  for (int r = threadIdx.x; r < len; r += JG_THREADS) {
    float x[TB];
#pragma unroll
    for (int i = 0; i < TB; ++i) x[i] = X[(size_t)i * pitch + r];
#pragma unroll 4
    for (int j = 0; j < TB; ++j) {
      float a0 = 0.f, a1 = 0.f;
#pragma unroll
      for (int i = 0; i < TB; i += 4) {
        const float4 c = *reinterpret_cast<const float4*>(&Jt[j][i]);
        a0 = fmaf(x[i], c.x, fmaf(x[i + 2], c.z, a0));
        a1 = fmaf(x[i + 1], c.y, fmaf(x[i + 3], c.w, a1));
      }
      put(j, r, a0 + a1);
    }
  }
}

// bits of max |a| over the CTA's share
__device__ __forceinline__ unsigned long long jg_max(const double* A, int64_t count, int64_t first,
                                                     int64_t step) {
  unsigned long long mx = 0ull;  // non-negative doubles order as their bits
  for (int64_t e = first; e < count; e += step) {
    const unsigned long long v = (unsigned long long)__double_as_longlong(fabs(A[e]));
    mx = v > mx ? v : mx;
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    const unsigned long long w = __shfl_xor_sync(0xffffffffu, mx, o);
    mx = w > mx ? w : mx;
  }
  return mx;
}
__device__ __forceinline__ double jg_scale(unsigned long long mx) {
  int ex = 0;
  frexp(__longlong_as_double((long long)mx), &ex);
  return ldexp(1.0, -ex);
}

template <int TB>
__global__ void __launch_bounds__(JG_THREADS, 1) jacobi_gram_cluster_kernel(const JgArgs p) {
  constexpr int B = TB / 2, C = JG_CLUSTER, steps = 2 * C - 1;
  extern __shared__ __align__(16) float jg_sm[];  // two buffers of TB x pitch
  __shared__ __align__(16) float Jt[TB][TB];
  __shared__ float G[TB][TB + 1];
  __shared__ float2 cs[B];
  __shared__ int2 pq[B];
  __shared__ unsigned long long mx_sh[C];
  __shared__ int cnt_sh[2][C];
  __shared__ float tm_sh[2][C], cm_sh[2][C];
  __shared__ int dst_sh[2], rot_sh;
  __shared__ float tmax_sh;
  cg::cluster_group cl = cg::this_cluster();
  const int rank = (int)cl.block_rank(), tid = threadIdx.x;
  const int n = p.n, pitch = p.pitch;
  const size_t half = (size_t)TB * pitch;

  // power-of-two scale: max |a| < 1
  if (tid < C) mx_sh[tid] = 0ull;
  if (tid == 0) {
    rot_sh = 0;
    tmax_sh = 0.f;
  }
  __syncthreads();
  {
    const unsigned long long mx = jg_max(p.A, (int64_t)n * n, (int64_t)rank * JG_THREADS + tid,
                                         (int64_t)C * JG_THREADS);
    if ((tid & 31) == 0) atomicMax(&mx_sh[rank], mx);
  }
  cl.sync();
  if (tid < C && tid != rank) mx_sh[tid] = *cl.map_shared_rank(&mx_sh[tid], tid);
  cl.sync();
  unsigned long long mx = 0ull;
  for (int r = 0; r < C; ++r) mx = mx_sh[r] > mx ? mx_sh[r] : mx;
  if (rank == 0 && tid == 0) *p.amax = mx;
  const double sc = jg_scale(mx);
  {
    int b0, b1;
    rr_pair(0, rank, 2 * C, b0, b1);
    for (int e = tid; e < TB * pitch; e += JG_THREADS) {
      const int j = e / pitch, i = e % pitch;
      const int col = (j < B ? b0 : b1) * B + j % B;
      jg_sm[e] = (col < n && i < n) ? (float)(p.A[(int64_t)col * n + i] * sc) : 0.f;
    }
  }
  __syncthreads();

  float cmax_prev = 0.f;
  int sweep = 0, cur = 0;
  for (; sweep < p.max_sweeps; ++sweep) {
    int rot = 0;
    float tmax = 0.f, cmax = 0.f;
    const float floor2 = sweep > 0 ? p.floor * p.floor * cmax_prev : 3.0e38f;
    for (int step = 0; step < steps; ++step) {
      const float* X = jg_sm + (size_t)cur * half;
      // where this CTA's blocks go next
      if (tid < 32) {
        int b0, b1, a = -1, b = -1;
        rr_pair(step, rank, 2 * C, b0, b1);
        if (tid < C) rr_pair(step + 1 < steps ? step + 1 : 0, tid, 2 * C, a, b);
#pragma unroll
        for (int side = 0; side < 2; ++side) {
          const int blk = side ? b1 : b0;
          const unsigned ma = __ballot_sync(0xffffffffu, a == blk);
          const unsigned mb = __ballot_sync(0xffffffffu, b == blk);
          if (tid == 0) dst_sh[side] = ma ? 2 * (__ffs(ma) - 1) : 2 * (__ffs(mb) - 1) + 1;
        }
      }
      jg_gram<TB>(X, pitch, G);
      __syncthreads();
      if (step == 0 && tid < TB) cmax = fmaxf(cmax, G[tid][tid]);
      jg_rounds<TB>(G, Jt, cs, pq, step == 0, p.tol, floor2, rot, tmax);
      float* Jo = p.J + (((int64_t)sweep * steps + step) * C + rank) * TB * TB;
      for (int e = tid; e < TB * TB / 4; e += JG_THREADS)
        reinterpret_cast<float4*>(Jo)[e] = reinterpret_cast<const float4*>(&Jt[0][0])[e];
      float* dst[2];
#pragma unroll
      for (int side = 0; side < 2; ++side)
        dst[side] = cl.map_shared_rank(jg_sm, dst_sh[side] >> 1) + (size_t)(cur ^ 1) * half +
                    (size_t)(dst_sh[side] & 1) * B * pitch;
      jg_apply<TB>(X, pitch, pitch, Jt, [&](int j, int r, float v) {
        (j < B ? dst[0] + (size_t)j * pitch : dst[1] + (size_t)(j - B) * pitch)[r] = v;
      });
      cur ^= 1;
      cl.sync();
    }
    // rotations, angles and norms of the sweep over the cluster
    if (tid < 32) {
      for (int o = 16; o > 0; o >>= 1) {
        rot += __shfl_xor_sync(0xffffffffu, rot, o);
        tmax = fmaxf(tmax, __shfl_xor_sync(0xffffffffu, tmax, o));
        cmax = fmaxf(cmax, __shfl_xor_sync(0xffffffffu, cmax, o));
      }
      const int par = sweep & 1;
      if (tid < C) {
        *cl.map_shared_rank(&cnt_sh[par][rank], tid) = rot;
        *cl.map_shared_rank(&tm_sh[par][rank], tid) = tmax;
        *cl.map_shared_rank(&cm_sh[par][rank], tid) = cmax;
      }
    }
    cl.sync();
    int total = 0;
    float tall = 0.f;
    cmax_prev = 0.f;
    for (int r = 0; r < C; ++r) {
      total += cnt_sh[sweep & 1][r];
      tall = fmaxf(tall, tm_sh[sweep & 1][r]);
      cmax_prev = fmaxf(cmax_prev, cm_sh[sweep & 1][r]);
    }
    if (total == 0) break;
    if (sweep > 0 && tall <= p.tstop) break;
  }
  if (rank == 0 && tid == 0) {
    const int done = sweep < p.max_sweeps ? sweep + 1 : sweep;
    p.info[ST_SWEEPS32] = done;
    *p.nsteps = done * steps;
  }
}

// the grid form: CTA k takes block pair k of every step
template <int TB>
__global__ void __launch_bounds__(JG_THREADS, 1) jacobi_gram_grid_kernel(const JgArgs p) {
  constexpr int B = TB / 2;
  extern __shared__ __align__(16) float jg_sm[];  // TB x pitch
  __shared__ __align__(16) float Jt[TB][TB];
  __shared__ float G[TB][TB + 1];
  __shared__ float2 cs[B];
  __shared__ int2 pq[B];
  __shared__ int abort_sh;
  cg::grid_group grid = cg::this_grid();
  const int n = p.n, pitch = p.pitch, nblk = p.nblk, steps = nblk - 1;
  const int tid = threadIdx.x, rank = blockIdx.x;
  const int64_t gtid = (int64_t)blockIdx.x * JG_THREADS + tid, gth = (int64_t)gridDim.x * JG_THREADS;
  if (tid == 0) abort_sh = 0;
  if (gtid == 0) {
    *p.amax = 0ull;
    *p.abortf = 0;
  }
  if (gtid < JG_MAX_SWEEPS) {
    p.counts[gtid] = 0;
    p.cmax[gtid] = 0u;
    p.tmax[gtid] = 0u;
  }
  for (int64_t e = gtid; e < nblk; e += gth) p.bflag[e] = 0;
  grid.sync();
  {
    const unsigned long long mx = jg_max(p.A, (int64_t)n * n, gtid, gth);
    if ((tid & 31) == 0 && mx) atomicMax(p.amax, mx);
  }
  grid.sync();
  {
    const double sc = jg_scale(*p.amax);
    int b0, b1;
    rr_pair(0, rank, nblk, b0, b1);
    for (int e = tid; e < TB * pitch; e += JG_THREADS) {
      const int j = e / pitch, i = e % pitch;
      const int col = (j < B ? b0 : b1) * B + j % B;
      jg_sm[e] = (col < n && i < n) ? (float)(p.A[(int64_t)col * n + i] * sc) : 0.f;
    }
  }
  __syncthreads();
  int gstep = 0, sweep = 0;
  for (; sweep < p.max_sweeps; ++sweep) {
    int rot = 0;
    float tmax = 0.f, cmax = 0.f;
    const float floor2 = sweep > 0 ? p.floor * p.floor * __uint_as_float(p.cmax[sweep - 1]) : 3.0e38f;
    for (int step = 0; step < steps; ++step, ++gstep) {
      int b0, b1;
      rr_pair(step, rank, nblk, b0, b1);
      if (gstep > 0) {
        // the two blocks, once their previous owners have released them
        if (tid < 2 && !abort_sh) {
          const int* fl = p.bflag + (tid ? b1 : b0);
          uint64_t t0 = 0;
          int v;
          asm volatile("ld.acquire.gpu.global.b32 %0, [%1];" : "=r"(v) : "l"(fl) : "memory");
          if (v < gstep) asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t0));
          while (v < gstep) {
            if (*(volatile int*)p.abortf) {
              abort_sh = 1;
              break;
            }
            uint64_t t1;
            asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t1));
            if (t1 - t0 > JG_WAIT_NS) {
              abort_sh = 1;
              atomicExch(p.abortf, 1);
              break;
            }
            asm volatile("ld.acquire.gpu.global.b32 %0, [%1];" : "=r"(v) : "l"(fl) : "memory");
          }
        }
        __syncthreads();
        if (abort_sh) {  // report and do no more work; the barriers stay uniform
          if (tid == 0) atomicMax(&p.info[ST_FAIL], PLOM_NUM_TIMEOUT);
          __syncthreads();
          continue;
        }
        const int pv = pitch / 4;
        for (int e = tid; e < TB * pv; e += JG_THREADS) {
          const int j = e / pv, v = e % pv;
          const int col = (j < B ? b0 : b1) * B + j % B;
          reinterpret_cast<float4*>(jg_sm)[e] =
              __ldcg(reinterpret_cast<const float4*>(p.At + (int64_t)col * pitch) + v);
        }
        __syncthreads();
      }
      jg_gram<TB>(jg_sm, pitch, G);
      __syncthreads();
      if (step == 0 && tid < TB) cmax = fmaxf(cmax, G[tid][tid]);
      jg_rounds<TB>(G, Jt, cs, pq, step == 0, p.tol, floor2, rot, tmax);
      jg_apply<TB>(jg_sm, pitch, pitch, Jt, [&](int j, int r, float v) {
        p.At[(int64_t)((j < B ? b0 : b1) * B + j % B) * pitch + r] = v;
      });
      float* Jo = p.J + ((int64_t)gstep * (nblk / 2) + rank) * TB * TB;
      for (int e = tid; e < TB * TB / 4; e += JG_THREADS)
        reinterpret_cast<float4*>(Jo)[e] = reinterpret_cast<const float4*>(&Jt[0][0])[e];
      __syncthreads();
      if (tid == 0) {
        __threadfence();
        asm volatile("st.release.gpu.global.b32 [%0], %1;" ::"l"(p.bflag + b0), "r"(gstep + 1) : "memory");
        asm volatile("st.release.gpu.global.b32 [%0], %1;" ::"l"(p.bflag + b1), "r"(gstep + 1) : "memory");
      }
    }
    if (tid < 32) {
      for (int o = 16; o > 0; o >>= 1) {
        rot += __shfl_xor_sync(0xffffffffu, rot, o);
        tmax = fmaxf(tmax, __shfl_xor_sync(0xffffffffu, tmax, o));
        cmax = fmaxf(cmax, __shfl_xor_sync(0xffffffffu, cmax, o));
      }
      if (tid == 0) {
        if (rot) atomicAdd(&p.counts[sweep], rot);
        atomicMax(&p.tmax[sweep], __float_as_uint(tmax));
        atomicMax(&p.cmax[sweep], __float_as_uint(cmax));
      }
    }
    grid.sync();
    if (*(volatile int*)p.abortf) break;
    if (p.counts[sweep] == 0) break;
    if (sweep > 0 && __uint_as_float(p.tmax[sweep]) <= p.tstop) break;
  }
  if (gtid == 0) {
    const int done = sweep < p.max_sweeps ? sweep + 1 : sweep;
    p.info[ST_SWEEPS32] = done;
    *p.nsteps = done * steps;
  }
}

// V = J_1 J_2 ... row by row: a CTA holds `R` rows of V and takes them through the
// block pairs of every step, the next step's J arriving while one is applied.
// Out: V (n x n row-major).
template <int TB>
__global__ void __launch_bounds__(256) jacobi_rows_kernel(const float* __restrict__ J,
                                                          const int* __restrict__ nsteps, int n,
                                                          int nblk, int R, float* __restrict__ V) {
  constexpr int B = TB / 2, OUT = 4;  // outputs a thread forms at a time
  extern __shared__ __align__(16) float jr_sm[];
  const int pairs = nblk / 2, steps = nblk - 1, ncol = nblk * B;
  const int jsz = pairs * TB * TB;       // floats of J per step
  float* jb = jr_sm;                     // [2][jsz]
  float* v = jr_sm + 2 * (size_t)jsz;    // [R][ncol]
  const int tid = threadIdx.x, r0 = blockIdx.x * R;
  const int total = *nsteps;
  for (int e = tid; e < R * ncol; e += 256) v[e] = (r0 + e / ncol == e % ncol) ? 1.f : 0.f;
  auto fetch = [&](int s, int buf) {
    const float4* src = reinterpret_cast<const float4*>(J + (int64_t)s * jsz);
    const uint32_t dst = (uint32_t)__cvta_generic_to_shared(jb + (size_t)buf * jsz);
    for (int e = tid; e < jsz / 4; e += 256)
      asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst + 16 * e), "l"(src + e) : "memory");
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  if (total > 0) fetch(0, 0);
  for (int s = 0; s < total; ++s) {
    if (s + 1 < total) {
      fetch(s + 1, (s + 1) & 1);
      asm volatile("cp.async.wait_group 1;" ::: "memory");
    } else {
      asm volatile("cp.async.wait_group 0;" ::: "memory");
    }
    __syncthreads();
    const float* js = jb + (size_t)(s & 1) * jsz;
    // a thread takes all TB outputs of one row and pair: rows of a pair's J are
    // shared by the R threads next to each other
    for (int it = tid; it < R * pairs; it += 256) {
      const int k = it / R, r = it % R;
      int b0, b1;
      rr_pair(s % steps, k, nblk, b0, b1);
      float* x0 = v + (size_t)r * ncol + b0 * B;
      float* x1 = v + (size_t)r * ncol + b1 * B;
      float x[TB];
#pragma unroll
      for (int i = 0; i < B; ++i) {
        x[i] = x0[i];
        x[B + i] = x1[i];
      }
      const float* jk = js + (size_t)k * TB * TB;
#pragma unroll 2
      for (int j = 0; j < TB; j += OUT) {
        float a[OUT];
#pragma unroll
        for (int u = 0; u < OUT; ++u) {
          a[u] = 0.f;
#pragma unroll
          for (int i = 0; i < TB; i += 4) {
            const float4 c = *reinterpret_cast<const float4*>(jk + (j + u) * TB + i);
            a[u] = fmaf(x[i], c.x, fmaf(x[i + 1], c.y, fmaf(x[i + 2], c.z, fmaf(x[i + 3], c.w, a[u]))));
          }
        }
#pragma unroll
        for (int u = 0; u < OUT; ++u) (j + u < B ? x0[j + u] : x1[j + u - B]) = a[u];
      }
    }
    __syncthreads();
  }
  for (int e = tid; e < R * n; e += 256) {
    const int r = e / n, c = e % n;
    if (r0 + r < n) V[(int64_t)(r0 + r) * n + c] = v[(size_t)r * ncol + c];
  }
}

// ---------------------------------------------------------------------------
// host side
// ---------------------------------------------------------------------------
struct JgPlan {
  bool cluster;
  int TB, nblk, pitch, R;
  const void *kern, *rows;
  size_t smem, rows_smem;
};

template <int TB>
static void jg_kernels(JgPlan& pl) {
  pl.TB = TB;
  pl.kern = pl.cluster ? (const void*)jacobi_gram_cluster_kernel<TB>
                       : (const void*)jacobi_gram_grid_kernel<TB>;
  pl.rows = (const void*)jacobi_rows_kernel<TB>;
}

// Up to 512 columns the 16 CTAs of a cluster hold all of them (32 columns of 512
// values twice, 131 KiB); beyond, 8-column blocks with one CTA per pair.
static bool jg_plan(JgPlan& pl, int n) {
  if (n < 1 || n > 1600) return false;
  pl.pitch = (int)(cdiv(n, 128) * 128);
  pl.cluster = n <= 512;
  if (pl.cluster) {
    pl.nblk = 2 * JG_CLUSTER;
    switch ((int)std::max<int64_t>(2, cdiv(n, 64))) {
      case 2: jg_kernels<8>(pl); break;
      case 3: jg_kernels<12>(pl); break;
      case 4: jg_kernels<16>(pl); break;
      case 5: jg_kernels<20>(pl); break;
      case 6: jg_kernels<24>(pl); break;
      case 7: jg_kernels<28>(pl); break;
      default: jg_kernels<32>(pl); break;
    }
    pl.smem = (size_t)2 * pl.TB * pl.pitch * sizeof(float);
  } else {
    const int nb = (int)cdiv(n, 8);
    pl.nblk = std::max(2, nb + (nb & 1));
    jg_kernels<16>(pl);
    pl.smem = (size_t)16 * pl.pitch * sizeof(float);
    if (pl.nblk / 2 > num_sms()) return false;
  }
  // rows of V per CTA: two CTAs' worth of rows per SM at most, J twice beside them
  pl.R = (int)std::max<int64_t>(1, std::min<int64_t>(8, cdiv(n, num_sms())));
  pl.rows_smem = ((size_t)2 * (pl.nblk / 2) * pl.TB * pl.TB + (size_t)pl.R * pl.nblk * (pl.TB / 2)) *
                 sizeof(float);
  return pl.rows_smem <= 220 * 1024;
}

bool jacobi_gram_plan_ok(int n) {
  JgPlan pl;
  return jg_plan(pl, n);
}

bool jacobi_gram_usable(int n) {
  JgPlan pl;
  if (!jg_plan(pl, n)) return false;
  if (cudaFuncSetAttribute(pl.kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)pl.smem) !=
          cudaSuccess ||
      cudaFuncSetAttribute(pl.rows, cudaFuncAttributeMaxDynamicSharedMemorySize,
                           (int)pl.rows_smem) != cudaSuccess) {
    cudaGetLastError();
    return false;
  }
  bool ok = false;
  if (pl.cluster) {
    if (cudaFuncSetAttribute(pl.kern, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) == cudaSuccess) {
      cudaLaunchConfig_t cfg = {};
      cudaLaunchAttribute at[1];
      at[0].id = cudaLaunchAttributeClusterDimension;
      at[0].val.clusterDim.x = JG_CLUSTER;
      at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
      cfg.gridDim = dim3(JG_CLUSTER);
      cfg.blockDim = dim3(JG_THREADS);
      cfg.dynamicSmemBytes = pl.smem;
      cfg.attrs = at;
      cfg.numAttrs = 1;
      int nc = 0;
      ok = cudaOccupancyMaxActiveClusters(&nc, pl.kern, &cfg) == cudaSuccess && nc >= 1;
    }
  } else {
    int per = 0;
    ok = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, pl.kern, JG_THREADS, pl.smem) ==
             cudaSuccess &&
         per >= 1 && pl.nblk / 2 <= per * num_sms();
  }
  cudaGetLastError();
  return ok;
}

int jacobi_gram_f32(const double* A, int n, float tol, float floor_rel, float tstop, float* V,
                    unsigned long long* amax, int* info, Arena& ws, cudaStream_t st) {
  JgPlan pl;
  PLOM_REQUIRE(jg_plan(pl, n), PLOM_ERR_UNSUPPORTED, "jacobi: %d columns", n);
  JgArgs a = {};
  const int pairs = pl.nblk / 2, steps = pl.nblk - 1;
  a.J = ws.take<float>((size_t)JG_MAX_SWEEPS * steps * pairs * pl.TB * pl.TB);
  a.nsteps = ws.take<int>(1);
  if (!pl.cluster) {
    a.At = ws.take<float>((size_t)pl.nblk * (pl.TB / 2) * pl.pitch);
    a.bflag = ws.take<int>(pl.nblk);
    a.abortf = ws.take<int>(1);
    a.counts = ws.take<int>(JG_MAX_SWEEPS);
    a.cmax = ws.take<unsigned>(JG_MAX_SWEEPS);
    a.tmax = ws.take<unsigned>(JG_MAX_SWEEPS);
  }
  if (ws.measuring()) return PLOM_OK;
  PLOM_REQUIRE(!ws.overflow(), PLOM_ERR_WORKSPACE, "jacobi: workspace too small");
  a.A = A;
  a.n = n;
  a.b = pl.TB / 2;
  a.nblk = pl.nblk;
  a.pitch = pl.pitch;
  a.tol = tol;
  a.floor = floor_rel;
  a.tstop = tstop;
  a.max_sweeps = JG_MAX_SWEEPS;
  a.amax = amax;
  a.info = info;
  ProfScope prof("jacobi_svd_f32", st, 0.0, 4.0 * 3.0 * n * n, 2);
  void* args[] = {(void*)&a};
  if (pl.cluster) {
    cudaLaunchConfig_t cfg = {};
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = JG_CLUSTER;
    at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
    cfg.gridDim = dim3(JG_CLUSTER);
    cfg.blockDim = dim3(JG_THREADS);
    cfg.dynamicSmemBytes = pl.smem;
    cfg.stream = st;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    PLOM_CHECK_CUDA(cudaLaunchKernelExC(&cfg, pl.kern, args));
  } else {
    PLOM_CHECK_CUDA(cudaLaunchCooperativeKernel(pl.kern, dim3(pairs), dim3(JG_THREADS), args, pl.smem, st));
  }
  const float* J = a.J;
  const int* ns = a.nsteps;
  void* rargs[] = {(void*)&J, (void*)&ns, (void*)&n, (void*)&pl.nblk, (void*)&pl.R, (void*)&V};
  PLOM_CHECK_CUDA(cudaLaunchKernel(pl.rows, dim3((unsigned)cdiv(n, pl.R)), dim3(256), rargs,
                                   pl.rows_smem, st));
  return PLOM_OK;
}

}  // namespace plom
