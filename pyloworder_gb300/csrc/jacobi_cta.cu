// One-sided Jacobi SVD of small matrices held in shared memory for all of
// their sweeps: one CTA per problem, or one thread-block cluster whose CTAs
// exchange column blocks through distributed shared memory.
//
// The block kernels of dense.cu fetch 8 columns of A^T and of V from L2 for
// every 4 rounds of rotations and pay a grid barrier (or a flag) for it: 10 to
// 12 us a block step whatever the row length, so problems of up to a few
// hundred columns are bound by that latency (32 columns: 84 steps, 1,039 us).
// Here a round costs one CTA barrier: 32 lanes (or 8, 16) hold a column pair
// in registers from the dot product to the rotation, and the rotation
// parameters are derived by every lane, in double-float arithmetic.
// Measured, block kernels -> here (4,096-row inputs, to convergence): 32 real
// columns 1,061 -> 260 us, 64 1,603 -> 953, 128 4,413 -> 1,943; 64 complex
// problems of 31 columns 3,127 -> 711 us, of 63 12,073 -> 3,590.  What bounds it: a round's chain of dependent
// instructions (1,700 cycles with one warp per scheduler, double-float), from 48
// columns on the issue rate of one SM, and in a cluster the exchange (8,000 to
// 11,000 cycles a step).
//
//  one CTA (C = 1): every column lives in the CTA.  The pairs follow the
//    block-of-4 schedule of dense.cu's kernels, all block pairs of a step side
//    by side, so the accumulated rotations (and with them the phases of complex
//    singular vectors) are those of that schedule.
//  cluster of C: CTA k holds two blocks of b = ceil(n / 2C) columns and meets
//    every other block in 2C - 1 steps of b rounds; between steps the blocks
//    move one place round the circle (each CTA reads the ones it needs from
//    its neighbours' shared memory).
//
// Arithmetic: double-float rows with scaled rotations (column = d x stored row,
// x' = x - t (dq/dp) e^{-i phi} y, y' = y + t (dp/dq) e^{i phi} x, d' = c d).
#include <cooperative_groups.h>

#include <algorithm>
#include <mutex>
#include <type_traits>

#include "plom_common.cuh"
#include "plom_df.cuh"
#include "plom_jacobi.cuh"

namespace cg = cooperative_groups;

namespace plom {

constexpr int JC_MAX_SWEEPS = 40;
constexpr float JC_FOLD = 9.094947017729282e-13f;  // 2^-40: a smaller scale goes into its row

// ---------------------------------------------------------------------------
// arithmetic of a column pair.  Rows are vectors of 16 bytes (V): 2 double-float
// values or 1 complex one.
// ---------------------------------------------------------------------------
// double-float state of a column: squared norm (x < 0: recompute), scale and
// its inverse
struct DfState { float2 nrm, d, e; };

// t of the rotation that makes a pair with norms al, be and |dot| g orthogonal
// (FP32: every t gives an exactly orthogonal rotation, c is exact for it)
__device__ __forceinline__ float jc_tan(float diff, float g) {
  const float z = __fdividef(diff, 2.0f * g);
  const float az = fabsf(z);
  const float w = fmaf(z, z, 1.0f);
  return az > 1e18f ? __fdividef(0.5f, z) : copysignf(__fdividef(1.0f, az + w * rsqrtf(w)), z);
}
// a pair with squared norms al, be and |dot| g is rotated
__device__ __forceinline__ bool jc_above(float al, float be, float g, float tol) {
  return al > 0.f && be > 0.f && g > tol * (al * rsqrtf(al)) * (be * rsqrtf(be));
}
// c = (1 + t^2)^-1/2 to double-float accuracy
__device__ __forceinline__ float2 jc_cos(float t) {
  const float p = __fmul_rn(t, t);
  float2 x = fast_two_sum(1.0f, p);
  x.y += fmaf(t, t, -p);
  return df_rsqrt(x);
}
// carried norms al - t g and be + t g (a drop below 1/8 is recomputed) and the
// scales of the rotated pair
__device__ __forceinline__ void jc_carry(DfState& p, DfState& q, float2 al, float2 be, float2 g,
                                         float t) {
  const float2 tg = df_mulf(g, t);
  const float2 na = df_add2(al, make_float2(-tg.x, -tg.y)), nb = df_add2(be, tg);
  p.nrm = (na.x > 0.125f * al.x) ? na : make_float2(-1.f, 0.f);
  q.nrm = (nb.x > 0.125f * be.x) ? nb : make_float2(-1.f, 0.f);
  const float2 c = jc_cos(t);
  p.d = df_mul(p.d, c);
  q.d = df_mul(q.d, c);
  p.e = df_recip(p.d);
  q.e = df_recip(q.d);
}
template <int L>
__device__ __forceinline__ float2 df_lane_sum(float2 v) {
  v = fast_two_sum(v.x, v.y);
#pragma unroll
  for (int o = L / 2; o > 0; o >>= 1) {
    const float h = __shfl_xor_sync(0xffffffffu, v.x, o);
    const float l = __shfl_xor_sync(0xffffffffu, v.y, o);
    const float2 s = two_sum(v.x, h);
    v = fast_two_sum(s.x, s.y + (v.y + l));
  }
  return v;
}

struct ArDf {
  using V = float4;  // two double-float values
  using S = DfState;
  static constexpr int PER = 2;
  struct Dot { float2 g0, g1; };
  struct Rot { float2 tp, tqn; bool on; };  // x -= tp y, y -= tqn x
  __device__ static V zero() { return make_float4(0.f, 0.f, 0.f, 0.f); }
  __device__ static void clear(Dot& d) { d.g0 = d.g1 = make_float2(0.f, 0.f); }
  __device__ static void dot(Dot& d, V x, V y) {
    df_dot_acc(d.g0, make_float2(x.x, x.y), make_float2(y.x, y.y));
    df_dot_acc(d.g1, make_float2(x.z, x.w), make_float2(y.z, y.w));
  }
  __device__ static void sq(float2& s, V x) {
    df_dot_acc(s, make_float2(x.x, x.y), make_float2(x.x, x.y));
    df_dot_acc(s, make_float2(x.z, x.w), make_float2(x.z, x.w));
  }
  template <int L>
  __device__ static Rot params(const Dot& dt, DfState& p, DfState& q, float tol) {
    const float2 s = two_sum(dt.g0.x, dt.g1.x);
    float2 g = df_lane_sum<L>(make_float2(s.x, s.y + (dt.g0.y + dt.g1.y)));
    Rot r;
    r.on = false;
    const float2 al = p.nrm, be = q.nrm;
    g = df_mul(df_mul(p.d, q.d), g);
    const float sg = g.x < 0.f ? -1.f : 1.f;
    g = make_float2(fabsf(g.x), sg * g.y);
    if (!jc_above(al.x, be.x, g.x, tol)) return r;
    const float2 df = two_sum(be.x, -al.x);
    const float t = jc_tan(df.x + (df.y + (be.y - al.y)), g.x);
    r.on = true;
    r.tp = df_mulf(df_mul(q.d, p.e), t * sg);
    r.tqn = df_mulf(df_mul(p.d, q.e), -t * sg);
    jc_carry(p, q, al, be, g, t);
    return r;
  }
  __device__ static void rotate(V& x, V& y, const Rot& r) {
    const float2 x0 = make_float2(x.x, x.y), x1 = make_float2(x.z, x.w);
    const float2 y0 = make_float2(y.x, y.y), y1 = make_float2(y.z, y.w);
    const float2 a0 = df_fms(x0, r.tp, y0), a1 = df_fms(x1, r.tp, y1);
    const float2 b0 = df_fms(y0, r.tqn, x0), b1 = df_fms(y1, r.tqn, x1);
    x = make_float4(a0.x, a0.y, a1.x, a1.y);
    y = make_float4(b0.x, b0.y, b1.x, b1.y);
  }
  __device__ static V scale(V x, float2 f) {
    const float2 a = df_mul(make_float2(x.x, x.y), f), b = df_mul(make_float2(x.z, x.w), f);
    return make_float4(a.x, a.y, b.x, b.y);
  }
};

struct ArDfC {
  using V = float4;  // one complex double-float value: re hi, re lo, im hi, im lo
  using S = DfState;
  static constexpr int PER = 1;
  struct Dot { float2 g0, g1; };  // Re, Im of x^H y
  // x -= w y, y += v x with w = tp (er - i ei), v = tq (er + i ei)
  struct Rot { float2 wr, wi, nvr, vi; bool on; };
  __device__ static V zero() { return make_float4(0.f, 0.f, 0.f, 0.f); }
  __device__ static void clear(Dot& d) { d.g0 = d.g1 = make_float2(0.f, 0.f); }
  __device__ static void dot(Dot& d, V x, V y) {
    const float2 xr = make_float2(x.x, x.y), xi = make_float2(x.z, x.w);
    const float2 yr = make_float2(y.x, y.y), yi = make_float2(y.z, y.w);
    df_dot_acc(d.g0, xr, yr);
    df_dot_acc(d.g0, xi, yi);
    df_dot_acc(d.g1, xr, yi);
    df_dot_acc(d.g1, make_float2(-xi.x, -xi.y), yr);
  }
  __device__ static void sq(float2& s, V x) {
    df_dot_acc(s, make_float2(x.x, x.y), make_float2(x.x, x.y));
    df_dot_acc(s, make_float2(x.z, x.w), make_float2(x.z, x.w));
  }
  template <int L>
  __device__ static Rot params(const Dot& dt, DfState& p, DfState& q, float tol) {
    const float2 dd = df_mul(p.d, q.d);
    float2 gr = df_mul(dd, df_lane_sum<L>(dt.g0)), gi = df_mul(dd, df_lane_sum<L>(dt.g1));
    Rot r;
    r.on = false;
    const float2 al = p.nrm, be = q.nrm;
    // |g| and the phase with g brought next to 1 by a power of two (its
    // square would leave the FP32 range)
    const float mx = fmaxf(fabsf(gr.x), fabsf(gi.x));
    if (!(al.x > 0.f && be.x > 0.f) || !(mx > 1e-37f)) return r;
    const int ex = (int)(__float_as_uint(mx) >> 23);  // biased exponent, 4 ... 254
    const float up = __uint_as_float((uint32_t)(254 - ex) << 23);
    const float dn = __uint_as_float((uint32_t)ex << 23);
    gr = make_float2(gr.x * up, gr.y * up);
    gi = make_float2(gi.x * up, gi.y * up);
    const float2 g2 = df_add2(df_mul(gr, gr), df_mul(gi, gi));
    const float2 ig = df_rsqrt(g2);
    float2 g = df_mul(g2, ig);
    g = make_float2(g.x * dn, g.y * dn);
    if (!jc_above(al.x, be.x, g.x, tol)) return r;
    const float2 er = df_mul(gr, ig), ei = df_mul(gi, ig);
    const float2 df = two_sum(be.x, -al.x);
    const float t = jc_tan(df.x + (df.y + (be.y - al.y)), g.x);
    const float2 tp = df_mulf(df_mul(q.d, p.e), t), tq = df_mulf(df_mul(p.d, q.e), t);
    r.on = true;
    r.wr = df_mul(tp, er);
    r.wi = df_mul(make_float2(-tp.x, -tp.y), ei);
    r.nvr = df_mul(make_float2(-tq.x, -tq.y), er);
    r.vi = df_mul(tq, ei);
    jc_carry(p, q, al, be, g, t);
    return r;
  }
  __device__ static void rotate(V& x, V& y, const Rot& r) {
    const float2 xr = make_float2(x.x, x.y), xi = make_float2(x.z, x.w);
    const float2 yr = make_float2(y.x, y.y), yi = make_float2(y.z, y.w);
    const float2 nwi = make_float2(-r.wi.x, -r.wi.y), nvi = make_float2(-r.vi.x, -r.vi.y);
    const float2 ar = df_fms(df_fms(xr, r.wr, yr), nwi, yi);   // xr - wr yr + wi yi
    const float2 ai = df_fms(df_fms(xi, r.wr, yi), r.wi, yr);  // xi - wr yi - wi yr
    const float2 br = df_fms(df_fms(yr, r.nvr, xr), r.vi, xi); // yr + vr xr - vi xi
    const float2 bi = df_fms(df_fms(yi, r.nvr, xi), nvi, xr);  // yi + vr xi + vi xr
    x = make_float4(ar.x, ar.y, ai.x, ai.y);
    y = make_float4(br.x, br.y, bi.x, bi.y);
  }
  __device__ static V scale(V x, float2 f) { return ArDf::scale(x, f); }
};

// ---------------------------------------------------------------------------
struct JacCtaArgs {
  const double* A;   // batch x n x n (complex: interleaved), ld n
  int n, C, bs;      // columns, CTAs per problem, columns per block
  int nblk;          // blocks (even)
  int rows;          // columns held by a CTA (rows of its A^T and V)
  float tol;
  int trans;         // rotate the rows of A instead of its columns (real)
  const double* V0;  // n x n starting rotation product (real; null: the identity)
  // the rotated columns, V and their norms, for jacobi_out_kernel
  double *At, *Vt, *nrm2;
  unsigned long long* amax;  // [batch]
  int* info;
  int max_sweeps;
};

// slot k of the block pairs of `step`: the block on `side`
__device__ __forceinline__ int jc_block(int step, int k, int nblk, int side) {
  int a, b;
  rr_pair(step, k, nblk, a, b);
  return side ? b : a;
}

template <typename Ar, int L, int Q, int T>
__global__ void __launch_bounds__(T, 1) jacobi_cta_kernel(const JacCtaArgs p) {
  using V = typename Ar::V;
  using S = typename Ar::S;
  constexpr int CW = std::is_same<Ar, ArDfC>::value ? 2 : 1;
  constexpr int PV = L * Q;          // vectors per row
  constexpr int GROUPS = T / L;      // column pairs in flight
  extern __shared__ __align__(16) unsigned char jc_smem[];
  __shared__ unsigned long long mx_sh[16];
  __shared__ int cnt_sh[2][16];
  __shared__ int rot_sh, src_sh[2];
  cg::cluster_group cl = cg::this_cluster();
  const int n = p.n, C = p.C, bs = p.bs, nblk = p.nblk, steps = nblk - 1;
  const int rank = C > 1 ? (int)cl.block_rank() : 0;
  const int prob = blockIdx.x / C;
  const int ntask = C > 1 ? 1 : nblk / 2;  // block pairs of this CTA
  V* cA = reinterpret_cast<V*>(jc_smem);
  V* cV = cA + (size_t)p.rows * PV;
  S* st = reinterpret_cast<S*>(cV + (size_t)p.rows * PV);
  const int tid = threadIdx.x, grp = tid / L, l = tid % L;
  const double* A = p.A + (int64_t)prob * n * n * CW;

  // row of column j of a block, and its global column
  auto row_of = [&](int side, int blk, int j) { return C > 1 ? side * bs + j : blk * bs + j; };

  // ---- power-of-two scale: max |a| < 1
  {
    if (tid < 16) mx_sh[tid] = 0ull;
    if (tid == 0) rot_sh = 0;
    __syncthreads();
    unsigned long long mx = 0ull;
    for (int64_t e = (int64_t)rank * T + tid; e < (int64_t)n * n * CW; e += (int64_t)C * T) {
      const unsigned long long v = (unsigned long long)__double_as_longlong(fabs(A[e]));
      mx = v > mx ? v : mx;
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      const unsigned long long w = __shfl_xor_sync(0xffffffffu, mx, o);
      mx = w > mx ? w : mx;
    }
    if ((tid & 31) == 0) atomicMax(&mx_sh[rank], mx);
    __syncthreads();
    if (C > 1) {
      cl.sync();
      if (tid < C && tid != rank) mx_sh[tid] = *cl.map_shared_rank(&mx_sh[tid], tid);
      cl.sync();
      if (tid == 0)
        for (int r = 1; r < C; ++r) mx_sh[0] = mx_sh[r] > mx_sh[0] ? mx_sh[r] : mx_sh[0];
      __syncthreads();
    }
  }
  int ex = 0;
  frexp(__longlong_as_double((long long)mx_sh[0]), &ex);
  if (rank == 0 && tid == 0) p.amax[prob] = mx_sh[0];
  // ---- rows in: columns of A (rows of A when trans), V = I
#pragma unroll 2
  for (int e = tid; e < p.rows * PV; e += T) {
    const int r = e / PV, v = e % PV;
    const int col = C > 1 ? jc_block(0, rank, nblk, r / bs) * bs + r % bs : r;
    V a = Ar::zero(), q = Ar::zero();
    if (col < n) {
      float* af = reinterpret_cast<float*>(&a);
      float* qf = reinterpret_cast<float*>(&q);
#pragma unroll
      for (int u = 0; u < Ar::PER; ++u) {
        const int i = v * Ar::PER + u;
        if (i >= n) continue;
        const int64_t src = p.trans ? (int64_t)col * n + i : (int64_t)i * n + col;
        if constexpr (CW == 1) {
          const float2 s = df_split(ldexp(A[src], -ex));
          af[2 * u] = s.x;
          af[2 * u + 1] = s.y;
          if (p.V0) {
            const float2 v0 = df_split(p.V0[(int64_t)i * n + col]);
            qf[2 * u] = v0.x;
            qf[2 * u + 1] = v0.y;
          } else {
            qf[2 * u] = i == col ? 1.f : 0.f;
          }
        } else {
          const float2 re = df_split(ldexp(A[2 * src], -ex));
          const float2 im = df_split(ldexp(A[2 * src + 1], -ex));
          a = make_float4(re.x, re.y, im.x, im.y);
          q.x = i == col ? 1.f : 0.f;
        }
      }
    }
    cA[e] = a;
    cV[e] = q;
  }
  for (int r = tid; r < p.rows; r += T) {
    st[r].d = st[r].e = make_float2(1.f, 0.f);
    st[r].nrm = make_float2(-1.f, 0.f);
  }
  __syncthreads();

  // squared norms of every held column, exactly
  auto norms = [&]() {
    for (int r0 = 0; r0 < p.rows; r0 += GROUPS) {  // uniform trip count: warp shuffles inside
      const int r = r0 + grp;
      const V* x = cA + (size_t)(r < p.rows ? r : 0) * PV;
      float2 s = make_float2(0.f, 0.f);
#pragma unroll
      for (int q = 0; q < Q; ++q) Ar::sq(s, x[l + q * L]);
      s = df_lane_sum<L>(s);
      if (l == 0 && r < p.rows) st[r].nrm = df_mul(df_mul(st[r].d, st[r].d), s);
    }
  };

  int sweep = 0;
  for (; sweep < p.max_sweeps; ++sweep) {
    int myrot = 0;
    for (int step = 0; step < steps; ++step) {
      if (C > 1 && (sweep > 0 || step > 0)) {
        // ---- the blocks of this step from the CTAs that held them
        const int prev = step > 0 ? step - 1 : steps - 1;
        if (tid < 32) {
#pragma unroll
          for (int side = 0; side < 2; ++side) {
            const int want = jc_block(step, rank, nblk, side);
            int a = -1, b = -1;
            if (tid < C) rr_pair(prev, tid, nblk, a, b);
            const unsigned ma = __ballot_sync(0xffffffffu, a == want);
            const unsigned mb = __ballot_sync(0xffffffffu, b == want);
            if (tid == 0) src_sh[side] = ma ? 2 * (__ffs(ma) - 1) : 2 * (__ffs(mb) - 1) + 1;
          }
        }
        cl.sync();  // every CTA is done with its pairs (and src_sh is set)
        constexpr int NV = 2 * Q;  // vectors a thread moves (bs <= GROUPS)
        V buf[NV];
        S sbuf = S();
        const int cnt = 2 * bs * PV;
#pragma unroll
        for (int half = 0; half < 2; ++half) {
          V* base = half ? cV : cA;
#pragma unroll
          for (int u = 0; u < NV; ++u) {
            const int v = tid + u * T;
            if (v < cnt) {
              const int side = v / (bs * PV), off = v - side * bs * PV;
              const int s = src_sh[side];
              const V* src = cl.map_shared_rank(base, s >> 1) + (size_t)(s & 1) * bs * PV + off;
              buf[u] = *src;
            }
          }
          if (half == 0 && tid < 2 * bs) {
            const int s = src_sh[tid / bs];
            sbuf = cl.map_shared_rank(st, s >> 1)[(s & 1) * bs + tid % bs];
          }
          cl.sync();  // read by all: the slots may be overwritten
#pragma unroll
          for (int u = 0; u < NV; ++u) {
            const int v = tid + u * T;
            if (v < cnt) base[v] = buf[u];
          }
          if (half == 0 && tid < 2 * bs) st[tid] = sbuf;
        }
        __syncthreads();
      }
      if (step == 0) {
        norms();
        __syncthreads();
      }
      // ---- rounds: inside the blocks at a sweep's first step, then across
      const int be = bs + (bs & 1);
      const int nintra = step == 0 ? be - 1 : 0;
      // the block pair and first column of this group's (first) slot
      int cb0, cb1, cpk;
      {
        const int task = C > 1 ? rank : grp / bs;
        cpk = C > 1 ? grp : grp % bs;
        rr_pair(step, task < nblk / 2 ? task : 0, nblk, cb0, cb1);
      }
      for (int rd = 0; rd < nintra + bs; ++rd) {
        const bool intra = rd < nintra;
        const int per = intra ? be : bs;
        const int slots = ntask * per;
        for (int s0 = 0; s0 < slots; s0 += GROUPS) {
          const int slot = s0 + grp;
          int ra = 0, rc = 0;
          bool live = slot < slots;
          if (live) {
            int b0 = cb0, b1 = cb1, pk = cpk, ja, jc, sa = 0, sc = 1;
            if (intra || s0 > 0) {
              const int task = C > 1 ? rank : slot / per;
              pk = slot % per;
              rr_pair(step, task, nblk, b0, b1);
            }
            if (intra) {
              const int h = pk >= be / 2;
              if (C == 1) intra_pair(rd, pk & 1, ja, jc);
              else rr_pair(rd, pk % (be / 2), be, ja, jc);
              if (h) b0 = b1;
              else b1 = b0;
              sa = sc = h;
            } else {
              ja = pk;
              jc = pk + rd - nintra;
              if (jc >= bs) jc -= bs;
            }
            live = ja < bs && jc < bs && b0 * bs + ja < n && b1 * bs + jc < n;
            if (live) {
              ra = row_of(sa, b0, ja);
              rc = row_of(sc, b1, jc);
            }
          }
          V* xa = cA + (size_t)ra * PV + l;
          V* ya = cA + (size_t)rc * PV + l;
          V x[Q], y[Q];
#pragma unroll
          for (int q = 0; q < Q; ++q) {
            x[q] = xa[q * L];
            y[q] = ya[q * L];
          }
          S sp = st[ra], sq = st[rc];
          V* xv = cV + (size_t)ra * PV + l;
          V* yv = cV + (size_t)rc * PV + l;
          {
            // a scale below 2^-40 goes into its row first (rare)
            const bool fa = live && sp.d.x < JC_FOLD, fb = live && sq.d.x < JC_FOLD;
            if (fa || fb) {
#pragma unroll
              for (int q = 0; q < Q; ++q) {
                if (fa) {
                  xa[q * L] = x[q] = Ar::scale(x[q], sp.d);
                  xv[q * L] = Ar::scale(xv[q * L], sp.d);
                }
                if (fb) {
                  ya[q * L] = y[q] = Ar::scale(y[q], sq.d);
                  yv[q * L] = Ar::scale(yv[q * L], sq.d);
                }
              }
              if (fa) sp.d = sp.e = make_float2(1.f, 0.f);
              if (fb) sq.d = sq.e = make_float2(1.f, 0.f);
            }
          }
          typename Ar::Dot dt;
          Ar::clear(dt);
#pragma unroll
          for (int q = 0; q < Q; ++q) Ar::dot(dt, x[q], y[q]);
          typename Ar::Rot r;
          {
            const bool need = live && (sp.nrm.x < 0.f || sq.nrm.x < 0.f);
            if (__any_sync(0xffffffffu, need)) {
              float2 a2 = make_float2(0.f, 0.f), b2 = a2;
#pragma unroll
              for (int q = 0; q < Q; ++q) {
                Ar::sq(a2, x[q]);
                Ar::sq(b2, y[q]);
              }
              a2 = df_lane_sum<L>(a2);
              b2 = df_lane_sum<L>(b2);
              if (sp.nrm.x < 0.f) sp.nrm = df_mul(df_mul(sp.d, sp.d), a2);
              if (sq.nrm.x < 0.f) sq.nrm = df_mul(df_mul(sq.d, sq.d), b2);
            }
            r = Ar::template params<L>(dt, sp, sq, p.tol);
            r.on = r.on && live;
          }
          if (r.on) {
#pragma unroll
            for (int q = 0; q < Q; ++q) {
              Ar::rotate(x[q], y[q], r);
              xa[q * L] = x[q];
              ya[q * L] = y[q];
              V a = xv[q * L], b = yv[q * L];
              Ar::rotate(a, b, r);
              xv[q * L] = a;
              yv[q * L] = b;
            }
          }
          if (live && l == 0) {
            st[ra] = sp;
            st[rc] = sq;
            myrot += r.on ? 1 : 0;
          }
        }
        __syncthreads();
      }
    }
    // ---- rotations of the sweep over the problem
    if (l == 0) {
      if (myrot) atomicAdd(&rot_sh, myrot);
    }
    __syncthreads();
    const int par = sweep & 1;
    if (tid < C) {
      int* dc = C > 1 ? cl.map_shared_rank(&cnt_sh[par][rank], tid) : &cnt_sh[par][0];
      *dc = rot_sh;
    }
    if (C > 1) cl.sync();
    else __syncthreads();
    int total = 0;
    for (int r = 0; r < C; ++r) total += cnt_sh[par][r];
    __syncthreads();
    if (tid == 0) rot_sh = 0;
    __syncthreads();
    if (total == 0) break;
  }

  // ---- out (the CTA holds the blocks of the last step)
  if (tid == 0 && rank == 0) {
    atomicMax(&p.info[ST_SWEEPS], sweep + 1);
    if (sweep >= p.max_sweeps) atomicMax(&p.info[ST_FAIL], PLOM_NUM_JACOBI);
  }
  norms();
  __syncthreads();
  const int len = n * CW;
  for (int e = tid; e < p.rows * len; e += T) {
    const int r = e / len, i = e % len;
    const int col = C > 1 ? jc_block(steps - 1, rank, nblk, r / bs) * bs + r % bs : r;
    if (col >= n) continue;
    const double d = df_val(st[r].d);
    const float2* a = reinterpret_cast<const float2*>(cA + (size_t)r * PV);
    const float2* v = reinterpret_cast<const float2*>(cV + (size_t)r * PV);
    p.At[((int64_t)prob * n + col) * len + i] = df_val(a[i]) * d;
    p.Vt[((int64_t)prob * n + col) * len + i] = df_val(v[i]) * d;
    if (i == 0) {
      double s = df_val(st[r].nrm);
      if (!(st[r].nrm.x > 1e-28f)) {  // near the end of the FP32 range: in FP64
        s = 0.0;
        for (int k = 0; k < len; ++k) {
          const double x = df_val(a[k]) * d;
          s = fma(x, x, s);
        }
      }
      p.nrm2[(int64_t)prob * n + col] = s;
    }
  }
  if (C > 1) cl.sync();  // no CTA leaves while a neighbour may read it
}

// S (descending), U and V^H from the rotated columns a_j, V's columns and the
// squared norms: one block per column.  A = Ub S Vb^H with Ub = a_j / sigma_j and
// Vb = v_j; trans: those of A^T, so U = Vb, V^T = Ub^T.
__global__ void __launch_bounds__(128) jacobi_out_kernel(const double* __restrict__ At,
                                                         const double* __restrict__ Vt,
                                                         const double* __restrict__ nrm2, int n,
                                                         int cw, int trans,
                                                         const unsigned long long* __restrict__ amax,
                                                         double* __restrict__ S,
                                                         double* __restrict__ U,
                                                         double* __restrict__ VH) {
  const int j = blockIdx.x;
  const int64_t b = blockIdx.y, rl = (int64_t)n * cw;
  __shared__ int part[4];
  const double* nb = nrm2 + b * n;
  const double sj = nb[j];
  int rank = 0;
  for (int k = threadIdx.x; k < n; k += 128) {
    const double sk = nb[k];
    rank += (sk > sj) || (sk == sj && k < j);
  }
  rank = warp_sum(rank);
  if ((threadIdx.x & 31) == 0) part[threadIdx.x >> 5] = rank;
  __syncthreads();
  const int k = part[0] + part[1] + part[2] + part[3];
  int ex = 0;
  frexp(__longlong_as_double((long long)amax[b]), &ex);
  const double sg = sqrt(sj);
  if (threadIdx.x == 0) S[b * n + k] = ldexp(sg, ex);
  const double f = sg > 0.0 ? 1.0 / sg : 0.0;
  const double* a = At + (b * n + j) * rl;
  const double* v = Vt + (b * n + j) * rl;
  double* Ub = U + b * n * rl;
  double* Vb = VH + b * n * rl + k * rl;
  for (int i = threadIdx.x; i < n; i += 128) {
    if (cw == 1) {
      const double ui = a[i] * f, vi = v[i];
      Ub[(int64_t)i * n + k] = trans ? vi : ui;
      Vb[i] = trans ? ui : vi;
    } else {
      Ub[(int64_t)i * rl + 2 * k] = a[2 * i] * f;
      Ub[(int64_t)i * rl + 2 * k + 1] = a[2 * i + 1] * f;
      Vb[2 * i] = v[2 * i];
      Vb[2 * i + 1] = -v[2 * i + 1];
    }
  }
}

// ---------------------------------------------------------------------------
// host side
// ---------------------------------------------------------------------------
// CTAs per problem, lanes per pair, vectors per lane, threads
struct JcPlan {
  int C, bs, nblk, rows, L, Q, T;
  const void* kern;
  size_t smem;
};

template <typename Ar, int L, int Q, int T>
static void jc_set(JcPlan& pl) {
  pl.L = L;
  pl.Q = Q;
  pl.T = T;
  pl.kern = (const void*)jacobi_cta_kernel<Ar, L, Q, T>;
  pl.smem = (size_t)pl.rows * (2 * L * Q * 16 + sizeof(typename Ar::S));
}

static void jc_blocks(JcPlan& pl, int n, int C) {
  pl.C = C;
  if (C == 1) {  // the block-of-4 schedule, every block in the CTA
    pl.bs = 4;
    const int nb = (n + 3) / 4;
    pl.nblk = std::max(2, nb + (nb & 1));
    pl.rows = n;
  } else {
    pl.bs = (n + 2 * C - 1) / (2 * C);
    pl.nblk = 2 * C;
    pl.rows = 2 * pl.bs;
  }
}

// Where the lines lie (double-float, real): one CTA issues n^2/2 pairs of 75 FP32
// instructions a row and a sweep, which passes the latency of a round (~0.3 us)
// near 64 columns; from there on the columns are spread over 4, 8 and 16 SMs.
// Complex problems (SPOD: one per frequency, tens of them) take one CTA each
// while A^H and V fit in its shared memory (83 columns).
static bool jc_plan(JcPlan& pl, int n, int cplx) {
  if (cplx) {
    if (n > 80) return false;
    jc_blocks(pl, n, 1);
    if (n <= 16) jc_set<ArDfC, 8, 2, 64>(pl);
    else if (n <= 24) jc_set<ArDfC, 8, 3, 128>(pl);
    else if (n <= 32) jc_set<ArDfC, 8, 4, 128>(pl);
    else if (n <= 48) jc_set<ArDfC, 8, 6, 192>(pl);
    else if (n <= 64) jc_set<ArDfC, 8, 8, 256>(pl);
    else jc_set<ArDfC, 8, 10, 320>(pl);
    return true;
  }
  if (n <= 64) {
    jc_blocks(pl, n, 1);
    if (n <= 16) jc_set<ArDf, 8, 1, 64>(pl);
    else if (n <= 32) jc_set<ArDf, 8, 2, 128>(pl);
    else if (n <= 48) jc_set<ArDf, 8, 3, 192>(pl);
    else jc_set<ArDf, 8, 4, 256>(pl);
    return true;
  }
  if (n <= 96) {
    jc_blocks(pl, n, 4);
    jc_set<ArDf, 16, 3, 192>(pl);
  } else if (n <= 128) {
    jc_blocks(pl, n, 8);
    jc_set<ArDf, 32, 2, 256>(pl);
  } else if (n <= 192) {
    jc_blocks(pl, n, 16);
    jc_set<ArDf, 32, 3, 192>(pl);
  } else if (n <= 256) {
    jc_blocks(pl, n, 16);
    jc_set<ArDf, 32, 4, 256>(pl);
  } else {
    return false;
  }
  return true;
}

// kernel attributes, and whether clusters of the plan's size can be resident
// (asked once per kernel and device)
static bool jc_ready(const JcPlan& pl) {
  struct Key {
    const void* k;
    int C, dev;
    size_t smem;
    bool ok;
  };
  static std::mutex mu;
  static Key seen[64];
  static int nseen = 0;
  int dev = 0;
  cudaGetDevice(&dev);
  std::lock_guard<std::mutex> lock(mu);
  for (int i = 0; i < nseen; ++i)
    if (seen[i].k == pl.kern && seen[i].C == pl.C && seen[i].dev == dev && seen[i].smem >= pl.smem)
      return seen[i].ok;
  bool ok = cudaFuncSetAttribute(pl.kern, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 (int)pl.smem) == cudaSuccess;
  if (ok && pl.C > 8)
    ok = cudaFuncSetAttribute(pl.kern, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) ==
         cudaSuccess;
  if (ok && pl.C > 1) {
    cudaLaunchConfig_t cfg = {};
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = pl.C;
    at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
    cfg.gridDim = dim3(pl.C);
    cfg.blockDim = dim3(pl.T);
    cfg.dynamicSmemBytes = pl.smem;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    int nc = 0;
    ok = cudaOccupancyMaxActiveClusters(&nc, pl.kern, &cfg) == cudaSuccess && nc >= 1;
  }
  cudaGetLastError();
  int slot = -1;  // a larger size of a known kernel replaces its entry
  for (int i = 0; i < nseen && slot < 0; ++i)
    if (seen[i].k == pl.kern && seen[i].C == pl.C && seen[i].dev == dev) slot = i;
  if (slot < 0 && nseen < 64) slot = nseen++;
  if (slot >= 0) seen[slot] = Key{pl.kern, pl.C, dev, pl.smem, ok};
  return ok;
}

static int jc_launch(const JcPlan& pl, const JacCtaArgs& a, int batch, cudaStream_t st) {
  cudaLaunchConfig_t cfg = {};
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = pl.C;
  at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
  cfg.gridDim = dim3((unsigned)(batch * pl.C));
  cfg.blockDim = dim3(pl.T);
  cfg.dynamicSmemBytes = pl.smem;
  cfg.stream = st;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  void* args[] = {(void*)&a};
  PLOM_CHECK_CUDA(cudaLaunchKernelExC(&cfg, pl.kern, args));
  return PLOM_OK;
}

bool jacobi_cta_usable(int n, int cplx) {
  JcPlan pl;
  return n >= 1 && jc_plan(pl, n, cplx) && jc_ready(pl);
}

int jacobi_cta(const double* A, int n, int batch, int cplx, int trans, double tol, double* At,
               double* Vt, double* nrm2, unsigned long long* amax, double* S, double* U,
               double* VH, int* info, cudaStream_t st, const double* V0) {
  JcPlan pl;
  PLOM_REQUIRE(jc_plan(pl, n, cplx), PLOM_ERR_UNSUPPORTED, "jacobi: %d columns", n);
  JacCtaArgs a = {};
  a.A = A;
  a.n = n;
  a.C = pl.C;
  a.bs = pl.bs;
  a.nblk = pl.nblk;
  a.rows = pl.rows;
  a.tol = (float)tol;
  a.trans = V0 ? 0 : trans;  // (from V0: A holds the rotated columns)
  a.V0 = V0;
  a.At = At;
  a.Vt = Vt;
  a.nrm2 = nrm2;
  a.amax = amax;
  a.info = info;
  a.max_sweeps = JC_MAX_SWEEPS;
  ProfScope prof("jacobi_svd_df", st, 0.0, 8.0 * 3.0 * n * n * batch * (cplx ? 2 : 1), 2);
  PLOM_TRY(jc_launch(pl, a, batch, st));
  jacobi_out_kernel<<<dim3((unsigned)n, (unsigned)batch), 128, 0, st>>>(
      At, Vt, nrm2, n, cplx ? 2 : 1, trans, amax, S, U, VH);
  PLOM_CHECK_LAUNCH();
  return PLOM_OK;
}

}  // namespace plom
