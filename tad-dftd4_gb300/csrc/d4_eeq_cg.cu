// EEQ solves of the precision form for structures beyond the one-CTA solver
// (N > 296) and few or small enough: conjugate gradients instead of a
// factorisation (eeq_cg_takes).
//
// The Coulomb matrix is positive definite and well conditioned (its smallest
// eigenvalues are the hardnesses, its largest grow as n^(2/3)): diagonally
// preconditioned CG gains six digits in 21 iterations at 1000 atoms and 29 at
// 4000, an iteration being one matrix-vector product, while the factorisation
// pays ~75 us per 128 columns in dependent steps.  The solve is the same
// refinement as before with CG in the factor's place: the residual b - A x in
// double-float (hi + lo matrix) is corrected by an FP32 solve, until it is
// where the factorisation left it (CgBars).
//
// One cooperative launch per solve.  A group of G CTAs shares a structure;
// each holds its rows of the matrix in shared memory when they fit and keeps
// the vectors r, s = A p and u = r / diag of the whole structure itself, so
// that an iteration exchanges nothing but the product (Chronopoulos and Gear's
// form, J. Comput. Appl. Math. 25, 153 (1989): the product is taken of u, one
// synchronisation): rows of A u to global memory, a barrier of the group, and
// every CTA updates its copies with the same arithmetic in the same order.
// Bound by the barrier and the L2 round trips of the exchange.
//
// Measured, charges / adjoint, against the factorisation (d4_eeq_big.cu):
// 997 atoms 1113 / 178 -> 226 / 188 us; the rule below has other sizes.  Of an
// iteration's 8200 cycles there, 2700 go to the barrier, 1450 to the product,
// 1480 to reading the exchanged rows and 2500 to the updates and reductions.
#include <float.h>
#include <math_constants.h>

#include "d4_common.cuh"
#include "d4_group.cuh"
#include "d4_kernels.cuh"

namespace d4 {

namespace {

// Threads per CTA: reductions and barriers cost per warp, the product of many
// rows wants more of them.  256 against 512 threads, charges / adjoint in us by
// rows per CTA: 8 (1 x 300) 139 / 102 and 148 / 109, 8 (1 x 997) 223 / 167 and
// 251 / 186, 11 (4 x 400) 173 / 125 and 174 / 123, 14 (1 x 2000) 404 / 329 and
// 392 / 302, 57 (16 x 512) 293 / 227 and 266 / 192.
constexpr int CG_FEW = 256, CG_MANY = 512, CG_FEW_ROWS = 10;
constexpr float CG_TOL = 1e-10f;     // max |b - A x| that converges
constexpr float CG_GAIN = 1e-12f;    // of (r, r / diag) per FP32 solve
constexpr float CG_LAST = 1e-10f;    // of it: FP32 may be at its end
constexpr int CG_OUTER = 16;         // refinements at most
constexpr int CG_INNER = 500;        // iterations of one FP32 solve at most
constexpr size_t CG_SMEM = 200 * 1024;

// Rows of A u (and residuals) in turn: two buffers, alternating, so that a CTA
// that is ahead does not overwrite what another still reads.
__device__ __forceinline__ float *cg_exchange(const Ctx &c, int b, int par) {
  return (par ? c.w.eeq_Y : c.w.eeq_V) + (size_t)b * 2 * c.N;
}
// Barrier counters, one per structure, in the room of the factorisation's
// panel operands (cleared by cg_rhs_kernel).
__device__ __forceinline__ unsigned *cg_counter(const Ctx &c, int b) {
  return reinterpret_cast<unsigned *>(c.w.eeq_P) + b;
}

struct CgSmem {
  __align__(16) float red[2][4][CG_MANY / 32];  // [turn][value][warp]
  int dead;
};

// Sums (or maxima from index NS on) of V values over the NT threads of the CTA,
// the same in all threads.  The buffers alternate, so one synchronisation is
// enough.
template <int NT, int V, int NS>
__device__ __forceinline__ void cg_reduce(float (&v)[V], CgSmem &sm, int &turn) {
#pragma unroll
  for (int q = 0; q < V; ++q) v[q] = q < NS ? warp_sumf(v[q]) : warp_maxf(v[q]);
  const int warp = threadIdx.x >> 5;
  turn ^= 1;
  if ((threadIdx.x & 31) == 0)
#pragma unroll
    for (int q = 0; q < V; ++q) sm.red[turn][q][warp] = v[q];
  __syncthreads();
#pragma unroll
  for (int q = 0; q < V; ++q) {
    const float4 *r = reinterpret_cast<const float4 *>(sm.red[turn][q]);
    float a = 0.f;  // (the maxima are of absolute values)
#pragma unroll
    for (int w = 0; w < NT / 128; ++w) {
      const float4 x = r[w];
      a = q < NS ? a + ((x.x + x.y) + (x.z + x.w))
                 : fmaxf(a, fmaxf(fmaxf(x.x, x.y), fmaxf(x.z, x.w)));
    }
    v[q] = a;
  }
}

__device__ __forceinline__ dfl cg_acc_prod(dfl acc, float h, float lo, float2 x) {
  const float p = h * x.x;
  const float e = fmaf(h, x.y, fmaf(lo, x.x, fmaf(h, x.x, -p)));
  const dfl s = df_two_sum(acc.hi, p);
  return {s.hi, acc.lo + (s.lo + e)};
}

__device__ __forceinline__ dfl cg_warp_sum(dfl a) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    const float oh = __shfl_xor_sync(0xffffffffu, a.hi, o);
    const float ol = __shfl_xor_sync(0xffffffffu, a.lo, o);
    const dfl s = df_two_sum(a.hi, oh);
    a = df_fast(s.hi, s.lo + (a.lo + ol));
  }
  return a;
}

// The factorisation's corrections overshoot CG_TOL: they leave 1e-11 (charges; what
// the residuals of a double-float solution resolve) and 1e-13 (adjoint).  So
// that these solves leave no more, one more correction follows where the first
// residual below CG_TOL is above ``goal``, and a correction after the first solve
// ends at ``end``, not at CG_TOL.  Residuals of charges / adjoint, ending at a
// quarter of CG_TOL and now: 997 atoms 1.8e-11 / 2.5e-11 and 7.8e-12 / 8e-14, 16000
// (d4_eeq_dcg.cu) 2.1e-11 / 2.4e-11 and 7.8e-12 / 1e-13, for 4 % of such calls' time.
//
// The adjoint's right-hand side is as large or small as the energies' weights make
// it.  It is solved times the power of two ``sc`` that brings its largest entry to
// ``top`` in [1, 2), so that no product of two residuals leaves FP32's range, and the
// bars follow it: those above for entries up to 1, relative beyond, and never
// above what the factorisation left of a small one (2e-7).
struct CgBars {
  float tol, goal, end;
};
__device__ __forceinline__ CgBars cg_charge_bars() { return {CG_TOL, 1.2e-11f, 9e-12f}; }
__device__ __forceinline__ CgBars cg_adjoint_bars(float sc, float top) {
  const float one = fmaxf(sc, top);
  return {CG_TOL * one, fminf(3e-13f * one, 2e-7f * top), fminf(1e-13f * one, 5e-8f * top)};
}

__host__ __device__ inline int cg_pad(int m) { return (m + 3) & ~3; }
// floats of the vectors of NR right-hand sides and of R rows of solution
__host__ __device__ inline size_t cg_vec_floats(int m, int nr, int R) {
  return (size_t)(3 * nr + 1) * cg_pad(m) + (size_t)nr * R * 4;
}

}  // namespace

// Right-hand sides as double-floats (compact order), zero solutions, barrier
// counters.
__global__ void cg_rhs_kernel(Ctx c, int adjoint) {
  const int b = blockIdx.y, N = c.N;
  const int k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k == 0) *cg_counter(c, b) = 0u;
  if (k < EEQ_BIG_REFINE) c.w.eeq_res[b * EEQ_BIG_REFINE + k] = 0u;  // empty structures
  if (k >= c.w.n_real[b]) return;
  const size_t ia = (size_t)b * N + c.w.ridx[(size_t)b * N + k], o = (size_t)b * 2 * N + k;
  dfl v;
  if (adjoint) {
    v = df_from(c.w.dEdq[ia]);
  } else {
    const int z = c.w.z[ia];
    const double cq = c.w.cnq[ia];
    v = df_from(-c.tab.eeq_chi[z] + c.tab.eeq_kcn[z] * (cq > 0.0 ? sqrt(cq) : 0.0));
    c.w.eeq_B[o + N] = make_float2(1.f, 0.f);
    c.w.eeq_X[o + N] = make_float2(0.f, 0.f);
  }
  c.w.eeq_B[o] = make_float2(v.hi, v.lo);
  c.w.eeq_X[o] = make_float2(0.f, 0.f);
}

// X = A^-1 B for NR right-hand sides of every structure.  ROWS: a CTA's rows
// of the matrix in shared memory.
template <int NT, int NR, bool ROWS>
__global__ void __launch_bounds__(NT, 1) eeq_cg_kernel(Ctx c, int G, int groups) {
  extern __shared__ __align__(16) float s_dyn[];
  __shared__ CgSmem sm;
  const int N = c.N;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int rank = blockIdx.x % G;
  if (group_gave_up(c.w.status)) return;
  if (tid == 0) sm.dead = 0;
  int turn = 0;
  for (int b = blockIdx.x / G; b < c.B; b += groups) {
    const int m = c.w.n_real[b];
    if (m == 0) continue;
    const int ms = cg_pad(m);
    const int row0 = (int)((long long)rank * m / G), row1 = (int)((long long)(rank + 1) * m / G);
    const int R = row1 - row0, RS = (m + G - 1) / G;
    float *r = s_dyn, *s = r + NR * ms, *u = s + NR * ms, *dinv = u + NR * ms;
    float2 *x = reinterpret_cast<float2 *>(dinv + ms);  // [NR][RS] own rows of the solution
    float *p = reinterpret_cast<float *>(x + NR * RS);  // [NR][RS]
    float *d = p + NR * RS;                             // [NR][RS]
    float *rows = s_dyn + ((cg_vec_floats(m, NR, RS) + 3) & ~(size_t)3);
    const float *Hi = c.w.eeq_hi + (size_t)b * N * N, *Lo = c.w.eeq_lo + (size_t)b * N * N;
    const float2 *B = c.w.eeq_B + (size_t)b * 2 * N;
    float2 *X = c.w.eeq_X + (size_t)b * 2 * N;
    unsigned *counter = cg_counter(c, b);
    unsigned passed = 0;
    int par = 0;
    float res = 0.f;
    __syncthreads();  // the last structure's shared memory is free
    for (int k = tid; k < ms; k += NT) {
      dinv[k] = k < m ? 1.0f / Hi[(size_t)k * N + k] : 0.f;
#pragma unroll
      for (int q = 0; q < NR; ++q) r[q * ms + k] = k < m ? B[q * N + k].x : 0.f;
    }
    if (ROWS)
      for (int i = warp; i < R; i += (NT / 32))
        for (int k = lane; k < ms; k += 32)
          rows[(size_t)i * ms + k] = k < m ? Hi[(size_t)(row0 + i) * N + k] : 0.f;
    for (int t = tid; t < NR * RS; t += NT) x[t] = make_float2(0.f, 0.f);
    float sc = 1.f;
    CgBars bars = cg_charge_bars();
    if (NR == 1) {
      float top[1] = {0.f};
      bool finite = true;
      for (int k = tid; k < ms; k += NT) {
        top[0] = fmaxf(top[0], fabsf(r[k]));
        finite = finite && fabsf(r[k]) <= FLT_MAX;
      }
      if (__syncthreads_or(!finite)) {  // every entry of the solution depends on all of them
        for (int t = tid; t < R; t += NT) X[row0 + t] = make_float2(CUDART_NAN_F, 0.f);
        continue;
      }
      cg_reduce<NT, 1, 0>(top, sm, turn);
      sc = scale_to_one(top[0]);
      bars = cg_adjoint_bars(sc, top[0] * sc);
      for (int k = tid; k < ms; k += NT) r[k] *= sc;
    }
    __syncthreads();
    bool alive = true, below = false;
    for (int outer = 0;; ++outer) {
      // the FP32 solve A d = r, from u = r / diag, p = s = 0
      float g[NR], mx[NR], beta[NR], alpha[NR];
      {
        float v[2 * NR];
#pragma unroll
        for (int q = 0; q < 2 * NR; ++q) v[q] = 0.f;
        for (int k = tid; k < ms; k += NT)
#pragma unroll
          for (int q = 0; q < NR; ++q) {
            const float rv = r[q * ms + k], uv = dinv[k] * rv;
            u[q * ms + k] = uv;
            s[q * ms + k] = 0.f;
            v[q] = fmaf(rv, uv, v[q]);
            v[NR + q] = fmaxf(v[NR + q], fabsf(rv));
          }
        for (int t = tid; t < NR * RS; t += NT) p[t] = d[t] = 0.f;
        cg_reduce<NT, 2 * NR, NR>(v, sm, turn);
#pragma unroll
        for (int q = 0; q < NR; ++q) {
          g[q] = v[q];
          mx[q] = v[NR + q];
          beta[q] = alpha[q] = 0.f;
        }
      }
      res = mx[0];
      if (NR == 2) res = fmaxf(res, mx[NR - 1]);
      if (res <= bars.goal || below || outer == CG_OUTER) break;
      below = res < bars.tol;  // (then this correction is the last)
      float stop[NR], g0[NR];
      bool on[NR];
#pragma unroll
      for (int q = 0; q < NR; ++q) {
        g0[q] = g[q];
        stop[q] = CG_GAIN * g[q];
        on[q] = mx[q] > bars.goal;
      }
      const float end = outer == 0 ? 0.f : bars.end;
      for (int it = 0; it < CG_INNER; ++it) {
        // own rows of A u
        float *w = cg_exchange(c, b, par);
        for (int i = warp; i < R; i += (NT / 32)) {
          float a[NR];
#pragma unroll
          for (int q = 0; q < NR; ++q) a[q] = 0.f;
          if (ROWS) {
            const float4 *h4 = reinterpret_cast<const float4 *>(rows + (size_t)i * ms);
            for (int k = lane; k < ms / 4; k += 32) {
              const float4 h = h4[k];
#pragma unroll
              for (int q = 0; q < NR; ++q) {
                const float4 v = reinterpret_cast<const float4 *>(u + q * ms)[k];
                a[q] = fmaf(h.x, v.x, fmaf(h.y, v.y, fmaf(h.z, v.z, fmaf(h.w, v.w, a[q]))));
              }
            }
          } else {
            const float *h = Hi + (size_t)(row0 + i) * N;
            const int whole = (N & 3) == 0 ? m / 4 : 0;  // 16-byte rows: 16-byte loads
#pragma unroll 8
            for (int k = lane; k < whole; k += 32) {
              const float4 hv = reinterpret_cast<const float4 *>(h)[k];
#pragma unroll
              for (int q = 0; q < NR; ++q) {
                const float4 v = reinterpret_cast<const float4 *>(u + q * ms)[k];
                a[q] = fmaf(hv.x, v.x, fmaf(hv.y, v.y, fmaf(hv.z, v.z, fmaf(hv.w, v.w, a[q]))));
              }
            }
#pragma unroll 8
            for (int k = 4 * whole + lane; k < m; k += 32) {
              const float hv = h[k];
#pragma unroll
              for (int q = 0; q < NR; ++q) a[q] = fmaf(hv, u[q * ms + k], a[q]);
            }
          }
#pragma unroll
          for (int q = 0; q < NR; ++q) a[q] = warp_sumf(a[q]);
          if (lane < NR) __stcg(&w[lane * N + row0 + i], lane == 0 ? a[0] : a[NR - 1]);
        }
        alive = group_barrier(counter, (unsigned)G * ++passed, sm.dead, c.w.status);
        if (!alive) break;
        par ^= 1;
        // p = u + beta p (own rows), s = A u + beta s, (A u, u)
        float v[NR];
#pragma unroll
        for (int q = 0; q < NR; ++q) v[q] = 0.f;
        for (int t = tid; t < NR * R; t += NT) {
          const int q = NR == 2 && t >= R, i = t - q * R;
          p[q * RS + i] = fmaf(beta[q], p[q * RS + i], u[q * ms + row0 + i]);
        }
#pragma unroll 4
        for (int k = tid; k < m; k += NT)
#pragma unroll
          for (int q = 0; q < NR; ++q) {
            const float wv = __ldcg(&w[q * N + k]);
            v[q] = fmaf(wv, u[q * ms + k], v[q]);
            s[q * ms + k] = fmaf(beta[q], s[q * ms + k], wv);
          }
        cg_reduce<NT, NR, NR>(v, sm, turn);
        bool bad = false, definite = true;
#pragma unroll
        for (int q = 0; q < NR; ++q) {
          if (!on[q]) {
            alpha[q] = 0.f;
            continue;
          }
          const float den = it == 0 ? v[q] : v[q] - beta[q] * g[q] / alpha[q];
          // (p, A p): not positive definite, or FP32 at its end, where the residual
          // of a definite matrix is
          if (!(den > 0.f)) {
            bad = true;
            definite = definite && it > 0 && v[q] > 0.f && g[q] <= CG_LAST * g0[q];
          }
          alpha[q] = g[q] / den;
        }
        if (bad) {
          if (!definite) {
            if (tid == 0) set_status(c.w.status, D4_ERR_EEQ_SINGULAR);
            outer = CG_OUTER - 1;  // the next residual is the last
          }
          break;
        }
        // d += alpha p (own rows), r -= alpha s, u = r / diag
        for (int t = tid; t < NR * R; t += NT) {
          const int q = NR == 2 && t >= R, i = t - q * R;
          d[q * RS + i] = fmaf(alpha[q], p[q * RS + i], d[q * RS + i]);
        }
        float n[2 * NR];
#pragma unroll
        for (int q = 0; q < 2 * NR; ++q) n[q] = 0.f;
        for (int k = tid; k < m; k += NT)
#pragma unroll
          for (int q = 0; q < NR; ++q) {
            const float rv = fmaf(-alpha[q], s[q * ms + k], r[q * ms + k]);
            const float uv = dinv[k] * rv;
            r[q * ms + k] = rv;
            u[q * ms + k] = uv;
            n[q] = fmaf(rv, uv, n[q]);
            n[NR + q] = fmaxf(n[NR + q], fabsf(rv));
          }
        cg_reduce<NT, 2 * NR, NR>(n, sm, turn);
        bool more = false;
#pragma unroll
        for (int q = 0; q < NR; ++q) {
          beta[q] = on[q] ? n[q] / g[q] : 0.f;
          g[q] = n[q];
          on[q] = on[q] && n[q] > stop[q] && n[NR + q] > end;
          more |= on[q];
        }
        if (!more) break;
      }
      if (!alive) break;
      // x += d; the residual in double-float
      __syncthreads();
      for (int t = tid; t < NR * R; t += NT) {
        const int q = NR == 2 && t >= R, i = t - q * R;
        const float2 o = x[q * RS + i];
        const dfl v = df_add(dfl{o.x, o.y}, dfl{d[q * RS + i], 0.f});
        x[q * RS + i] = make_float2(v.hi, v.lo);
        __stcg(&X[q * N + row0 + i], make_float2(v.hi, v.lo));
      }
      alive = group_barrier(counter, (unsigned)G * ++passed, sm.dead, c.w.status);
      if (!alive) break;
      float2 *xs = reinterpret_cast<float2 *>(s);  // [NR][ms], over s and u
      for (int k = tid; k < m; k += NT)
#pragma unroll
        for (int q = 0; q < NR; ++q) xs[q * ms + k] = __ldcg(&X[q * N + k]);
      __syncthreads();
      float *w = cg_exchange(c, b, par);
      for (int i = warp; i < R; i += (NT / 32)) {
        const int row = row0 + i;
        dfl a[NR];
#pragma unroll
        for (int q = 0; q < NR; ++q) a[q] = dfl{0.f, 0.f};
        const float *h = ROWS ? rows + (size_t)i * ms : Hi + (size_t)row * N;
        const float *l = Lo + (size_t)row * N;
#pragma unroll 4
        for (int k = lane; k < m; k += 32) {
          const float hv = h[k], lv = l[k];
#pragma unroll
          for (int q = 0; q < NR; ++q) a[q] = cg_acc_prod(a[q], hv, lv, xs[q * ms + k]);
        }
#pragma unroll
        for (int q = 0; q < NR; ++q) {
          const dfl t = cg_warp_sum(a[q]);
          const float2 bv = B[q * N + row];
          const dfl v = df_add(dfl{bv.x * sc, bv.y * sc}, df_neg(t));
          if (lane == 0) __stcg(&w[q * N + row], v.hi);
        }
      }
      alive = group_barrier(counter, (unsigned)G * ++passed, sm.dead, c.w.status);
      if (!alive) break;
      par ^= 1;
      for (int k = tid; k < ms; k += NT)
#pragma unroll
        for (int q = 0; q < NR; ++q) r[q * ms + k] = k < m ? __ldcg(&w[q * N + k]) : 0.f;
      __syncthreads();
    }
    if (!alive) return;
    if (NR == 1)  // (the exchanged solution was the scaled one)
      for (int t = tid; t < R; t += NT) X[row0 + t] = make_float2(x[t].x / sc, x[t].y / sc);
    if (rank == 0 && tid < EEQ_BIG_REFINE)
      c.w.eeq_res[b * EEQ_BIG_REFINE + tid] = __float_as_uint(res / sc);
  }
}

namespace {

struct CgPlan {
  int G, groups;  // CTAs per structure, structures at a time
  size_t vec, full;  // shared memory without and with the matrix rows
};

CgPlan cg_plan(const Ctx &c, int nr) {
  const int nsm = sm_count();
  // all SMs shared by the batch, at least eight rows each
  CgPlan p;
  const int most = (c.N + 7) / 8;
  p.G = nsm / c.B < most ? nsm / c.B : most;
  if (p.G < 1) p.G = 1;
  p.groups = c.B * p.G <= nsm ? c.B : nsm / p.G;
  const int R = (c.N + p.G - 1) / p.G;
  p.vec = 4 * ((cg_vec_floats(c.N, nr, R) + 3) & ~(size_t)3);
  p.full = p.vec + 4 * (size_t)R * cg_pad(c.N);
  return p;
}

template <int NR>
bool launch_cg(const Ctx &c, cudaStream_t st) {
  if (c.flags & D4_FLAG_TEST_FALLBACK) return false;
  CgPlan p = cg_plan(c, NR);
  const bool rows = p.full <= CG_SMEM;
  const size_t smem = rows ? p.full : p.vec;
  Ctx cc = c;
  void *args[] = {&cc, &p.G, &p.groups};
  const bool few = (c.N + p.G - 1) / p.G <= CG_FEW_ROWS;
  auto pick = [&](auto *many_rows, auto *many, auto *few_rows, auto *few_) {
    return few ? reinterpret_cast<const void *>(rows ? few_rows : few_)
               : reinterpret_cast<const void *>(rows ? many_rows : many);
  };
  const void *f = pick(&eeq_cg_kernel<CG_MANY, NR, true>, &eeq_cg_kernel<CG_MANY, NR, false>,
                       &eeq_cg_kernel<CG_FEW, NR, true>, &eeq_cg_kernel<CG_FEW, NR, false>);
  ensure_smem_impl(f, smem);
  keep_error();  // (a refused launch of this kernel itself is no error of the call)
  if (cudaLaunchCooperativeKernel(f, dim3((unsigned)(p.G * p.groups)),
                                  dim3(few ? CG_FEW : CG_MANY), args, smem, st) != cudaSuccess) {
    cudaGetLastError();
    return false;
  }
  return true;
}

}  // namespace

// Whether conjugate gradients solve the batch: when every CTA holds its matrix
// rows in shared memory, or when all SMs share few structures whose matrices
// stay in L2.  Charges + adjoint against the factorisation, us: 1 x 300 atoms
// 253 / 597, 1 x 997 413 / 1291, 1 x 2000 731 / 2170, 1 x 4000 1822 / 3616, 16 x
// 512 470 / 931; but 1 x 6001 8032 / 5645 (matrix from HBM) and 160 x 320 3032 /
// 1803 (a CTA per structure, matrix from L2).
bool eeq_cg_takes(const Ctx &c) {
  if (eeq_small_fits(c.N)) return false;
  const CgPlan p = cg_plan(c, 2);
  if (p.full <= CG_SMEM) return true;
  return p.vec <= CG_SMEM && p.G >= 16 && (size_t)4 * c.B * c.N * c.N <= (size_t)96 << 20;
}

bool launch_eeq_cg(const Ctx &c, cudaStream_t st, bool adjoint) {
  cg_rhs_kernel<<<dim3((c.N + 255) / 256, c.B), 256, 0, st>>>(c, adjoint ? 1 : 0);
  if (!(adjoint ? launch_cg<1>(c, st) : launch_cg<2>(c, st))) return false;
  launch_eeq_big_finish(c, st, adjoint, true);
  return true;
}

}  // namespace d4
