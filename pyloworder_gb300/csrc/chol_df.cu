// Shifted Cholesky R^T R = G + s I and the triangular inverse W = R^-1 of the
// mixed form's Gram matrices, in one kernel and in double-float arithmetic.
//
// What bounds the n x n stage is latency: on GB300 an FP64 square root and
// division by one thread take over a microsecond, so factoring one 32 x 32
// diagonal block took 55 us, the inverse 28 us more for its own blocks and two
// launches for each doubling of its size.  Here
//  * the arithmetic is double-float (48 bits; the Gram's own partial sums are
//    double-float, and its entries carry the 22-bit operands' rounding): 12 FP32
//    instructions a multiply-add against 64 FP32 issue slots for an FP64 one, and
//    a square root or reciprocal costs an FP32 estimate and one Newton step;
//  * G + s I is first scaled on both sides by powers of two that bring its
//    diagonal into [1/4, 1), so every entry fits the FP32 range;
//  * the elimination runs on [G + s I | I]: step k's trailing update subtracts
//    R_ka^T [R_kc | Z_kq], and the right half ends as Z = R^-T, so the inverse
//    needs no pass and no barrier of its own;
//  * a diagonal block is eliminated with one CTA barrier per column: every
//    thread keeps 8 rows of one of the 64 columns of [S | P] in registers, the
//    pivot row goes round through shared memory unscaled, and each thread derives
//    the pivot's reciprocal itself.
// Blocks are 32 x 32.  One problem of more than 64 columns takes one cooperative
// launch (two grid barriers a block step: panel, trailing update with the next
// diagonal block); batches and small problems take one CTA per problem and CTA
// barriers only.
#include <cooperative_groups.h>

#include <algorithm>

#include "plom_common.cuh"
#include "plom_df.cuh"
#include "plom_kernels.cuh"

namespace cg = cooperative_groups;

namespace plom {

constexpr int CB = 32;           // block size
constexpr int CPITCH = CB + 2;   // float2 per shared row (16-byte aligned rows)
constexpr int CD_ROUNDS = 8;     // shift escalations
constexpr int CD_THREADS = 256;
constexpr int CD_NEAR_GROUPS = 8;

struct CholDf {
  const double* G;
  double *R, *W;
  float2 *Rs, *Zs;   // batch x np x np: scaled [R | Z]
  float2* Dt;        // batch x 32 x 32: R_kk^-1 of the current block step
  float* d;          // batch x np: powers of two
  double *trace, *shift;
  int *status;       // 0 pending, 1 done, 2 failed in this round, 3 bad input
  int *pending, *used;
  double* colsq;     // near-identity test (batch 1)
  int* info;
  int n, np, batch, solo;
  double rel0, relfail, near_tol;
};

// 32 x 32 tile of a float2 matrix (ld np), 2 x 16 bytes a thread
__device__ __forceinline__ void cd_load(const float2* M, int ld, int bi, int bj, float4 (&v)[2]) {
  const float4* p = reinterpret_cast<const float4*>(M + (int64_t)bi * CB * ld + bj * CB);
#pragma unroll
  for (int u = 0; u < 2; ++u) {
    const int e = threadIdx.x + CD_THREADS * u;
    v[u] = p[(int64_t)(e >> 4) * (ld / 2) + (e & 15)];
  }
}
__device__ __forceinline__ void cd_stage(float2 (*S)[CPITCH], const float4 (&v)[2]) {
#pragma unroll
  for (int u = 0; u < 2; ++u) {
    const int e = threadIdx.x + CD_THREADS * u;
    *reinterpret_cast<float4*>(&S[e >> 4][2 * (e & 15)]) = v[u];
  }
}
// (A^T B) at rows 2 ty, 2 ty + 1 and columns 2 tx, 2 tx + 1
__device__ __forceinline__ void cd_mm(float2 (*A)[CPITCH], float2 (*B)[CPITCH], float2 (&c)[2][2]) {
  const int ty = threadIdx.x >> 4, tx = threadIdx.x & 15;
  c[0][0] = c[0][1] = c[1][0] = c[1][1] = make_float2(0.f, 0.f);
#pragma unroll 4
  for (int q = 0; q < CB; ++q) {
    const float4 a = *reinterpret_cast<const float4*>(&A[q][2 * ty]);
    const float4 b = *reinterpret_cast<const float4*>(&B[q][2 * tx]);
    const float2 a0 = make_float2(a.x, a.y), a1 = make_float2(a.z, a.w);
    const float2 b0 = make_float2(b.x, b.y), b1 = make_float2(b.z, b.w);
    df_dot_acc(c[0][0], a0, b0);
    df_dot_acc(c[0][1], a0, b1);
    df_dot_acc(c[1][0], a1, b0);
    df_dot_acc(c[1][1], a1, b1);
  }
}

__global__ void __launch_bounds__(CD_THREADS) chol_df_kernel(const CholDf p) {
  cg::grid_group grid = cg::this_grid();
  __shared__ __align__(16) float2 A[CB][CPITCH];
  __shared__ __align__(16) float2 B[CB][CPITCH];
  __shared__ __align__(16) float2 row_sh[2][2 * CB];
  __shared__ float2 piv_sh[CB];
  __shared__ double red[8];
  __shared__ int flag_sh;
  const int tid = threadIdx.x, n = p.n, np = p.np, T = np / CB;
  const int64_t nn = (int64_t)n * n, pp = (int64_t)np * np;
  // problems and tasks of this CTA: in solo mode its own problem's, else all
  // CTAs share the tasks of every problem
  const int b_lo = p.solo ? blockIdx.x : 0, b_n = p.solo ? 1 : p.batch;
  const int t0 = p.solo ? 0 : blockIdx.x, ts = p.solo ? 1 : gridDim.x;
  auto barrier = [&]() {
    if (p.solo) __syncthreads();
    else grid.sync();
  };

  // ---- trace and initial shift
  for (int bb = t0; bb < b_n; bb += ts) {
    const int b = b_lo + bb;
    double s = 0.0;
    for (int i = tid; i < n; i += CD_THREADS) s += p.G[b * nn + (int64_t)i * n + i];
    s = warp_sum(s);
    if ((tid & 31) == 0) red[tid >> 5] = s;
    __syncthreads();
    if (tid == 0) {
      double t = 0.0;
      for (int w = 0; w < CD_THREADS / 32; ++w) t += red[w];
      p.trace[b] = t;
      p.shift[b] = p.rel0 * t / n;
      p.status[b] = (isfinite(t) && t > 0.0) ? 0 : 3;
    }
    __syncthreads();
  }
  if (!p.solo && blockIdx.x == 0 && tid < CD_ROUNDS) p.pending[tid] = 0;
  if (p.near_tol > 0.0 && p.batch == 1 && p.rel0 == 0.0) {
    // G = I + E with X = triu(E, 1) + diag(E) / 2 and every ||X e_j||^2 <= near_tol:
    // R = I + X is the factor of G + X^T X, and R^-1 = I - X + X^2 up to X^3
    const int rows_g = (n + CD_NEAR_GROUPS - 1) / CD_NEAR_GROUPS;
    const int cblocks = (n + CD_THREADS - 1) / CD_THREADS;
    for (int task = t0; task < cblocks * CD_NEAR_GROUPS; task += ts) {
      const int g = task / cblocks, j = (task % cblocks) * CD_THREADS + tid;
      if (j >= n) continue;
      float2 acc = make_float2(0.f, 0.f);
      const int i1 = min(min(n, (g + 1) * rows_g), j + 1);
      for (int i = g * rows_g; i < i1; ++i) {
        const double e = p.G[(int64_t)i * n + j];
        const float2 x = df_split(i == j ? 0.5 * (e - 1.0) : e);
        df_dot_acc(acc, x, x);
      }
      p.colsq[(int64_t)g * n + j] = df_val(acc);
    }
    barrier();
    int ok = 1;
    for (int j = tid; j < n; j += CD_THREADS) {
      double c = 0.0;
      for (int g = 0; g < CD_NEAR_GROUPS; ++g) c += p.colsq[(int64_t)g * n + j];
      if (!(c <= p.near_tol)) ok = 0;  // (a NaN fails the test)
    }
    if (__syncthreads_and(ok) && p.status[0] == 0) {
      float(*X1)[CB + 1] = reinterpret_cast<float(*)[CB + 1]>(&A[0][0]);
      float(*X2)[CB + 1] = reinterpret_cast<float(*)[CB + 1]>(&B[0][0]);
      auto xat = [&](int i, int j) -> double {
        if (i >= n || j >= n || i > j) return 0.0;
        const double g = p.G[(int64_t)i * n + j];
        return i == j ? 0.5 * (g - 1.0) : g;
      };
      for (int t = t0; t < T * T; t += ts) {
        const int a = t / T, c = t % T;
        float acc[4] = {0.f, 0.f, 0.f, 0.f};
        for (int k = a; k <= c; ++k) {  // (X^2)_ac
          __syncthreads();
          for (int e = tid; e < CB * CB; e += CD_THREADS) {
            X1[e >> 5][e & 31] = (float)xat(a * CB + (e >> 5), k * CB + (e & 31));
            X2[e >> 5][e & 31] = (float)xat(k * CB + (e >> 5), c * CB + (e & 31));
          }
          __syncthreads();
          for (int q = 0; q < CB; ++q) {
#pragma unroll
            for (int u = 0; u < 4; ++u)
              acc[u] = fmaf(X1[(tid >> 5) + 8 * u][q], X2[q][tid & 31], acc[u]);
          }
        }
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          const int i = a * CB + (tid >> 5) + 8 * u, j = c * CB + (tid & 31);
          if (i >= n || j >= n) continue;
          const double x = xat(i, j), one = i == j ? 1.0 : 0.0;
          p.R[(int64_t)i * n + j] = one + x;
          p.W[(int64_t)i * n + j] = i <= j ? one - x + (double)acc[u] : 0.0;
        }
      }
      if (blockIdx.x == 0 && tid == 0) atomicAdd(&p.info[ST_NEAR], 1);
      return;  // every CTA takes the same branch: no barrier follows
    }
  }
  barrier();

  // ---- diagonal block of step k: [S | P] with S = R_kk (symmetric, upper part
  // valid) and P = I; eliminated to [R_kk | R_kk^-T]
  auto diag_block = [&](int b, int k) {
    if (p.status[b] != 0) return;
    float2* Rb = p.Rs + b * pp;
    const float* db = p.d + (int64_t)b * np;
    const int c = tid & 63, g = tid >> 6;  // column of [S | P], rows g, g + 4, ...
    const bool isS = c < CB;
    const int64_t dg = (int64_t)k * CB;
    float2 v[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const int a = g + 4 * i;
      v[i] = isS ? Rb[(dg + a) * np + dg + c] : make_float2(a == c - CB ? 1.f : 0.f, 0.f);
    }
    const double floor_piv = p.rel0 == 0.0 ? p.relfail * p.trace[b] / n : 0.0;
    if (g == 0) row_sh[0][c] = v[0];
    __syncthreads();
    bool ok = true;
    for (int j = 0; j < CB; ++j) {
      const float2* rw = row_sh[j & 1];
      float2 d = rw[j];
      bool good = d.x > 0.f && isfinite(d.x);
      if (!good && p.rel0 == 0.0 && isfinite(d.x)) {
        // unshifted factorisation (a CholeskyQR pass after the first): a null
        // direction of G, e.g. an exact zero column of the tall matrix.  This
        // pivot alone is floored; a shift of the whole diagonal would bias
        // every other column
        const float dj = db[dg + j];
        d = df_split(floor_piv * (double)dj * (double)dj);
        good = d.x > 0.f;
      }
      if (!good) {  // the same value in every thread
        ok = false;
        break;
      }
      const float2 rp = df_recip(d);
      if (tid == 0) piv_sh[j] = d;
      const float2 y = rw[c];
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        const int a = g + 4 * i;
        if (a <= j) continue;  // (warp-uniform)
        const float2 u = df_mul(rw[a], rp);
        v[i] = df_fms(v[i], u, y);
        if (a == j + 1) row_sh[(j + 1) & 1][c] = v[i];
      }
      __syncthreads();
    }
    if (!ok) {
      __syncthreads();
      if (tid == 0) p.status[b] = 2;
      __syncthreads();
      return;
    }
    // row a scaled by pivot^-1/2: R_ac (c >= a) and Z_aq (q <= a)
    float2* Zb = p.Zs + b * pp;
    float2* Db = p.Dt + (int64_t)b * CB * CB;
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const int a = g + 4 * i;
      const float2 rs = df_rsqrt(piv_sh[a]);
      const float2 zero = make_float2(0.f, 0.f);
      if (isS) {
        // (a floored pivot's diagonal entry is the pivot, not the stored value)
        const float2 x = c == a ? df_mul(piv_sh[a], rs) : df_mul(v[i], rs);
        Rb[(dg + a) * np + dg + c] = c >= a ? x : zero;
      } else {
        const int q = c - CB;
        const float2 x = q <= a ? df_mul(v[i], rs) : zero;
        Zb[(dg + a) * np + dg + q] = x;
        Db[q * CB + a] = x;  // R_kk^-1
      }
    }
    __syncthreads();
  };

  int round = 0;
  for (; round < CD_ROUNDS; ++round) {
    // ---- scales, then Rs = D (G + s I) D (upper blocks), Zs = 0
    for (int64_t e = (int64_t)t0 * CD_THREADS + tid; e < (int64_t)b_n * np; e += (int64_t)ts * CD_THREADS) {
      const int64_t b = b_lo + e / np;
      const int j = (int)(e % np);
      float d = 1.f;
      if (j < n) {
        const double h = p.G[b * nn + (int64_t)j * n + j] + p.shift[b];
        int ex = 0;
        if (h > 0.0 && isfinite(h)) frexp(h, &ex);
        ex = (ex + ((ex > 0) ? 1 : 0)) / 2;  // ceil(ex / 2)
        d = ldexpf(1.f, max(-120, min(120, -ex)));
      }
      p.d[b * np + j] = d;
    }
    barrier();
    for (int64_t e = (int64_t)t0 * CD_THREADS + tid; e < (int64_t)b_n * pp; e += (int64_t)ts * CD_THREADS) {
      const int64_t b = b_lo + e / pp, r = e % pp;
      if (p.status[b] != 0) continue;
      const int i = (int)(r / np), j = (int)(r % np);
      p.Zs[b * pp + r] = make_float2(0.f, 0.f);
      if (i / CB > j / CB) continue;
      float2 v = make_float2(i == j ? 1.f : 0.f, 0.f);
      if (i < n && j < n) {
        // the diagonal blocks hold both triangles
        double h = p.G[b * nn + (i <= j ? (int64_t)i * n + j : (int64_t)j * n + i)];
        if (i == j) h += p.shift[b];
        v = df_split(h * (double)p.d[b * np + i] * (double)p.d[b * np + j]);
      }
      p.Rs[b * pp + r] = v;
    }
    barrier();
    for (int bb = t0; bb < b_n; bb += ts) diag_block(b_lo + bb, 0);
    barrier();
    for (int k = 0; k < T; ++k) {
      // ---- panel: R_kj (j > k) and Z_kq (q < k) times R_kk^-T from the left
      const int ntp = T - 1;
      for (int t = t0; t < ntp * b_n; t += ts) {
        const int b = b_lo + t / ntp;
        const int r = t % ntp;
        if (p.status[b] != 0) continue;
        float2* M = (r < k ? p.Zs : p.Rs) + b * pp;
        const int j = r < k ? r : r + 1;
        float4 va[2], vb[2];
        cd_load(M, np, k, j, vb);
        const float4* dsrc = reinterpret_cast<const float4*>(p.Dt + (int64_t)b * CB * CB);
        va[0] = dsrc[tid];
        va[1] = dsrc[tid + CD_THREADS];
        cd_stage(A, va);
        cd_stage(B, vb);
        __syncthreads();
        float2 c[2][2];
        cd_mm(A, B, c);
        const int ty = tid >> 4, tx = tid & 15;
#pragma unroll
        for (int u = 0; u < 2; ++u) {
          const float2 x = fast_two_sum(c[u][0].x, c[u][0].y), y = fast_two_sum(c[u][1].x, c[u][1].y);
          *reinterpret_cast<float4*>(&M[((int64_t)k * CB + 2 * ty + u) * np + j * CB + 2 * tx]) =
              make_float4(x.x, x.y, y.x, y.y);
        }
        __syncthreads();
      }
      if (k == T - 1) break;
      barrier();
      // ---- trailing update: R_ac -= R_ka^T R_kc (k < a <= c) and
      // Z_aq -= R_ka^T Z_kq (a > k, q <= k); the next diagonal block first
      const int w = T - 1 - k;
      const int per = w * (w + 1) / 2 + w * (k + 1);
      for (int t = t0; t < per * b_n; t += ts) {
        int b, r;
        if (t < b_n) {
          b = t;
          r = 0;
        } else {
          const int u = t - b_n;
          b = u / (per - 1);
          r = 1 + u % (per - 1);
        }
        b += b_lo;
        if (p.status[b] != 0) continue;
        const bool next = r == 0;
        int a, c;
        float2* M;
        const int nr = w * (w + 1) / 2;
        if (r < nr) {
          a = 0;
          while (r >= w - a) {
            r -= w - a;
            ++a;
          }
          c = a + r + k + 1;
          a += k + 1;
          M = p.Rs + b * pp;
        } else {
          a = k + 1 + (r - nr) / (k + 1);
          c = (r - nr) % (k + 1);
          M = p.Zs + b * pp;
        }
        float4 va[2], vb[2];
        cd_load(p.Rs + b * pp, np, k, a, va);
        cd_load(M, np, k, c, vb);
        const int ty = tid >> 4, tx = tid & 15;
        float4 old[2];
#pragma unroll
        for (int u = 0; u < 2; ++u)
          old[u] = *reinterpret_cast<const float4*>(&M[((int64_t)a * CB + 2 * ty + u) * np + c * CB + 2 * tx]);
        cd_stage(A, va);
        cd_stage(B, vb);
        __syncthreads();
        float2 m[2][2];
        cd_mm(A, B, m);
#pragma unroll
        for (int u = 0; u < 2; ++u) {
          const float2 x = df_add2(make_float2(old[u].x, old[u].y), make_float2(-m[u][0].x, -m[u][0].y));
          const float2 y = df_add2(make_float2(old[u].z, old[u].w), make_float2(-m[u][1].x, -m[u][1].y));
          *reinterpret_cast<float4*>(&M[((int64_t)a * CB + 2 * ty + u) * np + c * CB + 2 * tx]) =
              make_float4(x.x, x.y, y.x, y.y);
        }
        __syncthreads();
        if (next) diag_block(b, k + 1);
      }
      barrier();
    }
    barrier();
    // ---- outcome of the round
    if (p.solo) {
      const int b = b_lo, s = p.status[b];
      __syncthreads();
      if (s == 2) {
        if (tid == 0) {
          const double base = p.relfail * p.trace[b] / n;
          p.shift[b] = fmax(p.shift[b] * 100.0, base);
          p.status[b] = 0;
          atomicMax(p.used, round + 1);
        }
        __syncthreads();
        continue;
      }
      if (s == 0 && tid == 0) p.status[b] = 1;
      __syncthreads();
      break;
    }
    for (int b = blockIdx.x * CD_THREADS + tid; b < p.batch; b += gridDim.x * CD_THREADS) {
      const int s = p.status[b];
      if (s == 0) {
        p.status[b] = 1;
      } else if (s == 2) {
        const double base = p.relfail * p.trace[b] / n;
        p.shift[b] = fmax(p.shift[b] * 100.0, base);
        p.status[b] = 0;
        atomicAdd(&p.pending[round], 1);
        atomicMax(p.used, round + 1);
      }
    }
    barrier();
    if (p.pending[round] == 0) break;
  }
  // ---- out: R = Rs D^-1, W = D Zs^T
  for (int64_t e = (int64_t)t0 * CD_THREADS + tid; e < (int64_t)b_n * nn; e += (int64_t)ts * CD_THREADS) {
    const int64_t b = b_lo + e / nn, r = e % nn;
    const int i = (int)(r / n), j = (int)(r % n);
    const float* db = p.d + b * np;
    const bool up = i <= j;
    p.R[b * nn + r] = up ? df_val(p.Rs[b * pp + (int64_t)i * np + j]) * (double)(1.0f / db[j]) : 0.0;
    p.W[b * nn + r] = up ? df_val(p.Zs[b * pp + (int64_t)j * np + i]) * (double)db[i] : 0.0;
  }
  for (int bb = t0 * CD_THREADS + tid; bb < b_n; bb += ts * CD_THREADS) {
    const int s = p.status[b_lo + bb];
    if (s == 0 || s == 2) atomicMax(&p.info[ST_FAIL], PLOM_NUM_CHOLESKY);
    if (s == 3) atomicMax(&p.info[ST_FAIL], PLOM_NUM_NONFINITE);
  }
  if (tid == 0 && (p.solo || blockIdx.x == 0)) atomicMax(&p.info[ST_SHIFTS], *p.used);
}

int chol_inverse_df(const double* G, double* R, double* W, int n, int batch, double rel0,
                    double relfail, int* info, Arena& ws, cudaStream_t st, double near_tol) {
  CholDf p = {};
  const int T = (n + CB - 1) / CB;
  p.np = T * CB;
  const size_t pp = (size_t)p.np * p.np;
  p.Rs = ws.take<float2>(pp * batch);
  p.Zs = ws.take<float2>(pp * batch);
  p.Dt = ws.take<float2>((size_t)batch * CB * CB);
  p.d = ws.take<float>((size_t)batch * p.np);
  p.trace = ws.take<double>(batch);
  p.shift = ws.take<double>(batch);
  p.status = ws.take<int>(batch);
  p.used = ws.take<int>(1);
  p.pending = ws.take<int>(CD_ROUNDS);
  p.colsq = (batch == 1 && rel0 == 0.0 && near_tol > 0.0)
                ? ws.take<double>((size_t)CD_NEAR_GROUPS * n)
                : nullptr;
  if (ws.measuring() || n == 0 || batch == 0) return PLOM_OK;
  PLOM_REQUIRE(!ws.overflow(), PLOM_ERR_WORKSPACE, "chol: workspace too small");
  PLOM_REQUIRE(G && R && W && info, PLOM_ERR_ARG, "chol: null pointer");
  PLOM_CHECK_CUDA(cudaMemsetAsync(p.used, 0, sizeof(int), st));
  p.G = G;
  p.R = R;
  p.W = W;
  p.info = info;
  p.n = n;
  p.batch = batch;
  p.rel0 = rel0;
  p.relfail = relfail;
  p.near_tol = p.colsq ? near_tol : 0.0;
  // one CTA per problem when the blocks are few (3 tiles a step at 64 columns:
  // 2 us each, no more than a grid barrier) or the problems are many
  p.solo = T <= 2 || batch >= 16;
  ProfScope prof("chol_df", st, 2.0 * (double)n * n * n / 3.0 * batch, 24.0 * n * n * batch);
  if (p.solo) {
    chol_df_kernel<<<batch, CD_THREADS, 0, st>>>(p);
    PLOM_CHECK_LAUNCH();
    return PLOM_OK;
  }
  int64_t want = 1;
  for (int k = 0; k < T; ++k) {
    const int64_t w = T - 1 - k;
    want = std::max(want, (w * (w + 1) / 2 + w * (k + 1)) * batch);
  }
  // at most one CTA per SM: they share its FP32 pipe, and fewer CTAs make
  // each grid barrier cheaper
  const int blocks = (int)std::min<int64_t>(want, num_sms());
  void* args[] = {(void*)&p};
  PLOM_CHECK_CUDA(cudaLaunchCooperativeKernel((const void*)chol_df_kernel, dim3(blocks),
                                              dim3(CD_THREADS), args, 0, st));
  return PLOM_OK;
}

}  // namespace plom
