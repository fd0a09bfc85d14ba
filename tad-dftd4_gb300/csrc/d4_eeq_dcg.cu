// EEQ solves of the precision form for large structures in spatial order:
// deflated conjugate gradients over half of the matrix, instead of a
// factorisation (eeq_dcg_takes).
//
// What slows diagonally preconditioned CG down as structures grow are the few
// smooth, large-eigenvalue modes of the Coulomb matrix.  Blocks of 64
// consecutive atoms are compact in space (Z-order), so the piecewise constant
// vectors Z of the blocks (K <= 256 of them) hold those modes: CG on
// P A, P = 1 - A Z (Z^T A Z)^-1 Z^T, gains five digits in 14 iterations at 6000
// atoms and 17 at 16000, where plain CG takes 32 at 6000.  As in d4_eeq_cg.cu the
// FP32 solve is the inner one of a refinement whose residuals are taken in
// double-float.
//
// Measured at 16000 atoms, charges + adjoint: 22.0 (factorisation) -> 12.0 ms, of
// it 8.8 the solves (73 products), 1.7 the residuals, 1.0 the matrix, 0.4 Z^T A Z,
// its inverse and G.  A product takes 93 us
// with one right-hand side (5.5 TB/s of the half matrix), 122 with two; the rest
// of an iteration (two exchanges, three barriers) 12 to 14 us.
//
// An iteration is one product with A, bound by reading the matrix: only tiles
// on and below the diagonal are read, each for both of its products (rows from
// registers, columns through shared memory), and a tile's row is replaced by
// the next tile's as soon as it is used, so 64 KB per SM are in flight.  One
// cooperative launch per solve, one CTA per SM; a CTA owns a slice of the
// vectors (registers) and of G = A Z (Z^T A Z)^-1 (shared memory).  The
// product is taken of u - Z mu, mu = G^T u, which is P A u without forming (and
// cancelling) the smooth part of A u, and projected again: with either alone
// FP32 rounding keeps the deflated modes at 1e-4 of the right-hand side (16000
// atoms) or brings them back every ten iterations.  Chronopoulos and
// Gear's form of CG (J. Comput. Appl. Math. 25, 153 (1989)); deflation after
// Nicolaides (SIAM J. Numer. Anal. 24, 355 (1987)) in the form of Saad et al.
// (SIAM J. Sci. Comput. 21, 1909 (2000)).
#include "d4_common.cuh"
#include "d4_group.cuh"
#include "d4_kernels.cuh"

namespace d4 {

namespace {

constexpr int DC_BLOCK = 64;  // atoms per block vector
constexpr int DC_K = 256;     // blocks at most
constexpr int DC_TILE = EEQ_HALF_TILE;
constexpr int DC_THREADS = 512, DC_WARPS = DC_THREADS / 32, DC_ROWS = DC_TILE / DC_WARPS;
constexpr int DC_SLICE = DC_THREADS / 4;  // rows of a CTA's slice at most (four lanes each)
constexpr int DC_LDG = DC_K + 16;         // row stride of G in shared memory (no bank conflicts)
constexpr float DC_TOL = 1e-10f;          // max |b - A x| that converges
constexpr float DC_GAIN = 3e-9f;          // of (r, r / diag) per FP32 solve (1e-8 to 1e-9 alike;
                                          // 1e-11 takes 2 % more of a call of 16000 atoms)
constexpr float DC_LAST = 1e-8f;          // of it: FP32 may be at its end
constexpr float DC_FLOOR = 1e-14f;        // of (b, b / diag): FP32 rounding of r
constexpr int DC_ITS = 100;               // iterations of one FP32 solve at most

// Scratch: A Z and G in the room of the factor's block inverses, the rest in
// that of its panel operands.
struct DcArea {
  float *AZ, *G;              // [N][DC_K]
  float *A0, *Ai;             // [DC_K][DC_K] Z^T A Z and its inverse
  float *w[2], *u;            // [2][dc_pad(N)] (two products in turn)
  float *mu[2];               // [DC_COPIES][2][DC_K] G^T u (in turn)
  float *t[2];                // [2][DC_K] Z^T w (in turn)
  float *tr;                  // [EEQ_BIG_REFINE][2][DC_K] Z^T r of each solve's start
  float2 *dot;                // [ranks][2] partial (A u, u), (r, u)
  float4 *norm;               // [ranks][2] partial (r, u), max |r|, (b, b / diag)
  unsigned *counter;          // [EEQ_BIG_REFINE] barriers of each solve
  float *top;                 // [1] largest entry of the adjoint's right-hand side
};
constexpr size_t DC_RANKS = 512;
constexpr int DC_COPIES = 8;  // of the sums that every CTA adds to at once (same L2 lines)

// stride of a vector: whole tiles (u is zero beyond the structure)
__host__ __device__ inline size_t dc_pad(int N) {
  return (size_t)((N + DC_TILE - 1) / DC_TILE) * DC_TILE;
}
__host__ __device__ inline size_t dc_floats(int N) {
  return 2 * (size_t)DC_K * DC_K + 6 * dc_pad(N) +
         (4 + 4 * DC_COPIES + 2 * EEQ_BIG_REFINE) * DC_K + 12 * DC_RANKS + 64;
}
__host__ __device__ inline size_t dc_stride(int N) {  // bytes of panel operands per structure
  return 2 * (size_t)eeq_nblk(N) * EEQ_OPND_BLOCK;
}

__device__ __forceinline__ DcArea dc_area(const Ctx &c, int b) {
  const size_t NP = dc_pad(c.N);
  DcArea a;
  a.AZ = c.w.eeq_Xd + (size_t)b * eeq_nsb(c.N) * EEQ_SB * EEQ_SB;
  a.G = a.AZ + (size_t)c.N * DC_K;
  float *f = reinterpret_cast<float *>(c.w.eeq_P + b * dc_stride(c.N));
  a.A0 = f;
  a.Ai = a.A0 + DC_K * DC_K;
  a.w[0] = a.Ai + DC_K * DC_K;
  a.w[1] = a.w[0] + 2 * NP;
  a.u = a.w[1] + 2 * NP;
  a.mu[0] = a.u + 2 * NP;
  a.mu[1] = a.mu[0] + DC_COPIES * 2 * DC_K;
  a.t[0] = a.mu[1] + DC_COPIES * 2 * DC_K;
  a.t[1] = a.t[0] + 2 * DC_K;
  a.tr = a.t[1] + 2 * DC_K;
  a.dot = reinterpret_cast<float2 *>(a.tr + EEQ_BIG_REFINE * 2 * DC_K);
  a.norm = reinterpret_cast<float4 *>(a.dot + 2 * DC_RANKS);
  a.counter = reinterpret_cast<unsigned *>(a.norm + 2 * DC_RANKS);
  a.top = reinterpret_cast<float *>(a.counter + EEQ_BIG_REFINE);
  return a;
}

// The bars of a solve, as in d4_eeq_cg.cu (CgBars): the residual that converges, the
// one it aims at, and where a correction after the first solve ends.  top: the
// largest entry of the adjoint's right-hand side.
struct DcBars {
  float tol, goal, end;
};
__device__ __forceinline__ DcBars dc_bars(const Ctx &c, int b, int nr) {
  if (nr == 2) return {DC_TOL, 1.2e-11f, 9e-12f};
  const float top = *dc_area(c, b).top, one = fmaxf(1.f, top);
  return {DC_TOL * one, fminf(3e-13f * one, 2e-7f * top), fminf(1e-13f * one, 5e-8f * top)};
}

// Whether iteration ``it`` has nothing to do: the goal is reached, or the last one
// was the one that may follow a residual below ``tol``.  Its entry of eeq_res
// then repeats the last one's (dcg_rest_kernel).
__device__ __forceinline__ bool dc_skip(const Ctx &c, int b, int it, int nr) {
  if (it == 0) return false;
  const unsigned *res = c.w.eeq_res + b * EEQ_BIG_REFINE + it;
  const DcBars bars = dc_bars(c, b, nr);
  return __uint_as_float(res[-1]) <= bars.goal ||
         (it > 1 && __uint_as_float(res[-2]) < bars.tol);
}

__device__ __forceinline__ float4 dc_stream4(const float *p) {
  float4 v;
  asm volatile("ld.global.nc.L1::no_allocate.v4.f32 {%0, %1, %2, %3}, [%4];"
               : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w)
               : "l"(p));
  return v;
}

struct DcSmem {
  float G[DC_SLICE * DC_LDG];
  float z[2][2][DC_WARPS][DC_TILE];  // [turn][right-hand side][warp]: a tile's column sums
  float tb[2][DC_K], mu[2][DC_K], t[2][DC_K];  // Z^T b; G^T u; Z^T w
  float ui[2][DC_TILE];
  float x[2][DC_SLICE];
  float red[DC_WARPS][8];
  float4 sum[2];
  float2 dot[2];
  float y[2][4];
  int dead;
};

// w += A (u - Z mu), t += Z^T of it, over tiles t0 .. t1 - 1 of the lower triangle
// (row by row).  Warp v takes rows 8 v .. 8 v + 7 of a tile; VEC (rows 16-byte
// aligned): lane l columns 4 l .. 4 l + 3, else l, l + 32, l + 64, l + 96.
template <int NR, bool VEC>
__device__ __forceinline__ void dc_product(const float *__restrict__ Hi, int N, int m, int t0,
                                           int t1, const float *u, float *w, float *tc,
                                           DcSmem &sm) {
  if (t0 >= t1) return;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  auto col = [&](int J, int e) { return DC_TILE * J + (VEC ? 4 * lane + e : lane + 32 * e); };
  // Loads carry no condition, so that nothing waits for them before their use:
  // rows beyond the structure repeat the last one (u is zero there), columns
  // beyond it (last diagonal tile only) are cleared at their use.
  auto load_row = [&](float (&h)[4], int I, int J, int r) {
    const float *p = Hi + (size_t)min(DC_TILE * I + DC_ROWS * warp + r, m - 1) * N;
    if (VEC) {
      const float4 v = dc_stream4(p + min(col(J, 0), N - 4));
      h[0] = v.x, h[1] = v.y, h[2] = v.z, h[3] = v.w;
    } else {
#pragma unroll
      for (int e = 0; e < 4; ++e) h[e] = __ldg(p + min(col(J, e), m - 1));
    }
  };
  const size_t us = dc_pad(N);
  auto load_u = [&](float (&v)[NR][4], int J) {
#pragma unroll
    for (int q = 0; q < NR; ++q) {
      if (VEC) {
        const float4 x = __ldcg(reinterpret_cast<const float4 *>(u + q * us + col(J, 0)));
        v[q][0] = x.x, v[q][1] = x.y, v[q][2] = x.z, v[q][3] = x.w;
      } else {
#pragma unroll
        for (int e = 0; e < 4; ++e) v[q][e] = __ldcg(u + q * us + col(J, e));
      }
    }
  };
  auto minus_mu = [&](float (&v)[NR][4], int J) {
#pragma unroll
    for (int q = 0; q < NR; ++q)
#pragma unroll
      for (int e = 0; e < 4; ++e) v[q][e] -= sm.mu[q][2 * J + (VEC ? lane >> 4 : e >> 1)];
  };
  int I, J;
  tri_entry(t0, I, J);
  float h[DC_ROWS][4], uj[NR][4], y[DC_ROWS][NR];
#pragma unroll
  for (int r = 0; r < DC_ROWS; ++r) load_row(h[r], I, J, r);
  load_u(uj, J);
  minus_mu(uj, J);
  bool first = true;
  int turn = 0;
  for (int t = t0; t < t1; ++t) {
    if (first || J == 0) {  // a new row of tiles
      first = false;
      __syncthreads();
      if (tid < NR * DC_TILE) {
        const int q = tid / DC_TILE, k = tid % DC_TILE;
        const int row = DC_TILE * I + k;
        sm.ui[q][k] = row < m ? __ldcg(u + q * us + row) - sm.mu[q][row / DC_BLOCK] : 0.f;
      }
      __syncthreads();
#pragma unroll
      for (int r = 0; r < DC_ROWS; ++r)
#pragma unroll
        for (int q = 0; q < NR; ++q) y[r][q] = 0.f;
    }
    const bool diag = J == I, more = t + 1 < t1;
    const int In = diag ? I + 1 : I, Jn = diag ? 0 : J + 1;
    float un[NR][4], z[NR][4];
    load_u(un, more ? Jn : J);
#pragma unroll
    for (int q = 0; q < NR; ++q)
#pragma unroll
      for (int e = 0; e < 4; ++e) z[q][e] = 0.f;
    const bool edge = DC_TILE * (J + 1) > m;
#pragma unroll
    for (int r = 0; r < DC_ROWS; ++r) {
      if (edge) {
#pragma unroll
        for (int e = 0; e < 4; ++e) h[r][e] = col(J, e) < m ? h[r][e] : 0.f;
      }
#pragma unroll
      for (int q = 0; q < NR; ++q) {
        const float ui = sm.ui[q][DC_ROWS * warp + r];
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          y[r][q] = fmaf(h[r][e], uj[q][e], y[r][q]);
          z[q][e] = fmaf(h[r][e], ui, z[q][e]);
        }
      }
      if (more) load_row(h[r], In, Jn, r);
    }
    if (!diag) {  // the mirrored tile's product, summed over the warps
#pragma unroll
      for (int q = 0; q < NR; ++q) {
        float *o = sm.z[turn][q][warp];
        if (VEC) {
          *reinterpret_cast<float4 *>(o + 4 * lane) =
              make_float4(z[q][0], z[q][1], z[q][2], z[q][3]);
        } else {
#pragma unroll
          for (int e = 0; e < 4; ++e) o[lane + 32 * e] = z[q][e];
        }
      }
      __syncthreads();
      if (tid < NR * DC_TILE) {
        const int q = tid / DC_TILE, k = tid % DC_TILE, row = DC_TILE * J + k;
        float s = 0.f;
#pragma unroll
        for (int v = 0; v < DC_WARPS; ++v) s += sm.z[turn][q][v][k];
        atomicAdd(w + q * us + row, s);  // (J < I: row < m)
        s = warp_sumf(s);
        if (lane == 0) atomicAdd(tc + q * DC_K + row / DC_BLOCK, s);
      }
      turn ^= 1;
    }
    if (diag || !more) {  // the row of tiles ends
#pragma unroll
      for (int q = 0; q < NR; ++q) {
        const int row0 = DC_TILE * I + DC_ROWS * warp;
        float s = 0.f;
#pragma unroll
        for (int r = 0; r < DC_ROWS; ++r) {
          const float v = warp_sumf(y[r][q]);
          if (row0 + r < m) {
            if (lane == 0) atomicAdd(w + q * us + row0 + r, v);
            s += v;
          }
        }
        if (lane == 0 && row0 < m) atomicAdd(tc + q * DC_K + row0 / DC_BLOCK, s);
      }
    }
    I = In;
    J = Jn;
#pragma unroll
    for (int q = 0; q < NR; ++q)
#pragma unroll
      for (int e = 0; e < 4; ++e) uj[q][e] = un[q][e];
    if (more) minus_mu(uj, J);
  }
}

// Sums (max from index NS on) of the warps' values v over the CTA, for thread 0;
// all lanes of a warp enter.
template <int V, int NS>
__device__ __forceinline__ void dc_cta_sum(float (&v)[V], DcSmem &sm) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
#pragma unroll
  for (int q = 0; q < V; ++q) v[q] = q < NS ? warp_sumf(v[q]) : warp_maxf(v[q]);
  if (lane == 0)
#pragma unroll
    for (int q = 0; q < V; ++q) sm.red[warp][q] = v[q];
  __syncthreads();
  if (warp == 0) {
#pragma unroll
    for (int q = 0; q < V; ++q) {
      const float s = lane < DC_WARPS ? sm.red[lane][q] : 0.f;
      v[q] = q < NS ? warp_sumf(s) : warp_maxf(s);
    }
  }
}

}  // namespace

// A Z: sums of A over the columns of each block.  A CTA per pair of blocks on or
// below the diagonal: its row sums, and its column sums for the mirrored pair.
__global__ void __launch_bounds__(256) dcg_az_kernel(Ctx c) {
  constexpr int ROWS = DC_BLOCK / 8;  // of a warp
  __shared__ float s_col[8][DC_BLOCK];
  const int b = blockIdx.y, m = c.w.n_real[b], N = c.N;
  int I, J;
  tri_entry(blockIdx.x, I, J);
  if (DC_BLOCK * I >= m) return;
  const DcArea ar = dc_area(c, b);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int row0 = DC_BLOCK * I + ROWS * warp, l = DC_BLOCK * J + lane;
  const float *h = c.w.eeq_hi + (size_t)b * N * N;
  float a[ROWS][2], s[2] = {0.f, 0.f};
#pragma unroll
  for (int r = 0; r < ROWS; ++r)
#pragma unroll
    for (int e = 0; e < 2; ++e) {
      const bool ok = row0 + r < m && l + 32 * e < m;
      a[r][e] = ok ? __ldg(h + (size_t)(row0 + r) * N + l + 32 * e) : 0.f;
    }
#pragma unroll
  for (int r = 0; r < ROWS; ++r) {
    s[0] += a[r][0];
    s[1] += a[r][1];
    const float v = warp_sumf(a[r][0] + a[r][1]);
    if (lane == 0 && row0 + r < m) ar.AZ[(size_t)(row0 + r) * DC_K + J] = v;
  }
  if (I != J) {  // (J < I: whole columns)
    s_col[warp][lane] = s[0];
    s_col[warp][lane + 32] = s[1];
    __syncthreads();
    if (threadIdx.x < DC_BLOCK) {
      float v = 0.f;
#pragma unroll
      for (int w = 0; w < 8; ++w) v += s_col[w][threadIdx.x];
      ar.AZ[(size_t)(DC_BLOCK * J + threadIdx.x) * DC_K + I] = v;
    }
  } else {
    const int K = (m + DC_BLOCK - 1) / DC_BLOCK;
    for (int r = row0; r < min(row0 + ROWS, m); ++r)
      for (int k = K + lane; k < DC_K; k += 32) ar.AZ[(size_t)r * DC_K + k] = 0.f;
  }
}

// Z^T A Z, a CTA per block.
__global__ void __launch_bounds__(DC_K) dcg_a0_kernel(Ctx c) {
  const int b = blockIdx.y, m = c.w.n_real[b], k = blockIdx.x, l = threadIdx.x;
  if (DC_BLOCK * k >= m) return;
  const DcArea ar = dc_area(c, b);
  const int r1 = min(m, DC_BLOCK * (k + 1));
  float s = 0.f;
  for (int r = DC_BLOCK * k; r < r1; ++r) s += ar.AZ[(size_t)r * DC_K + l];
  ar.A0[k * DC_K + l] = s;
}

// (Z^T A Z)^-1 by sweeping every pivot (Gauss-Jordan elimination of a symmetric
// matrix, which stays symmetric; no pivoting, it is positive definite), one CTA
// per structure: thread (y, x) of 32 x 32 holds entries (y + 32 i, x + 32 j),
// j <= i, in registers.  One barrier and 36 FMAs per thread and pivot.
__global__ void __launch_bounds__(1024) dcg_inverse_kernel(Ctx c) {
  __shared__ float s_row[2][DC_K];
  const int b = blockIdx.x, m = c.w.n_real[b];
  if (m == 0) return;
  const DcArea ar = dc_area(c, b);
  const int K = (m + DC_BLOCK - 1) / DC_BLOCK;
  const int x = threadIdx.x & 31, y = threadIdx.x >> 5;
  constexpr int Q = DC_K / 32;
  float v[Q * (Q + 1) / 2];
  auto at = [](int i, int j) { return i * (i + 1) / 2 + j; };
#pragma unroll
  for (int i = 0; i < Q; ++i)
#pragma unroll
    for (int j = 0; j <= i; ++j) {
      const int r = y + 32 * i, l = x + 32 * j;
      v[at(i, j)] = r < K && l < K ? ar.A0[r * DC_K + l] : (r == l ? 1.f : 0.f);
    }
  bool bad = false;
#pragma unroll
  for (int pa = 0; pa < Q; ++pa) {
    if (32 * pa >= K) break;
#pragma unroll 1
    for (int pt = 0; pt < 32; ++pt) {
      float *row = s_row[pt & 1];  // entries (p, .) = (., p) of pivot p = 32 pa + pt
      if (y == pt)
#pragma unroll
        for (int j = 0; j <= pa; ++j) row[x + 32 * j] = v[at(pa, j)];
      if (x == pt)
#pragma unroll
        for (int i = pa + 1; i < Q; ++i) row[y + 32 * i] = v[at(i, pa)];
      __syncthreads();
      const float piv = row[32 * pa + pt], inv = 1.0f / piv;
      bad |= !(piv > 0.f);
      float rj[Q];
#pragma unroll
      for (int j = 0; j < Q; ++j) rj[j] = row[x + 32 * j];
#pragma unroll
      for (int i = 0; i < Q; ++i) {
        const float f = row[y + 32 * i] * inv;
        const bool prow = i == pa && y == pt;
#pragma unroll
        for (int j = 0; j <= i; ++j) {
          const bool pcol = j == pa && x == pt;
          float &a = v[at(i, j)];
          a = prow ? (pcol ? -inv : rj[j] * inv) : (pcol ? f : fmaf(-f, rj[j], a));
        }
      }
    }
  }
  if (bad && threadIdx.x == 0) set_status(c.w.status, D4_ERR_EEQ_SINGULAR);
#pragma unroll
  for (int i = 0; i < Q; ++i)
#pragma unroll
    for (int j = 0; j <= i; ++j) {
      const int r = y + 32 * i, l = x + 32 * j;
      const float a = r < K && l < K ? -v[at(i, j)] : 0.f;
      ar.Ai[r * DC_K + l] = a;
      if (i != j) ar.Ai[l * DC_K + r] = a;
    }
}

// G = A Z (Z^T A Z)^-1: 32 rows per CTA, a column per thread.
constexpr int DG_ROWS = 32;
__global__ void __launch_bounds__(DC_K) dcg_g_kernel(Ctx c) {
  __shared__ __align__(16) float s_az[DG_ROWS][DC_K];
  const int b = blockIdx.y, m = c.w.n_real[b], r0 = blockIdx.x * DG_ROWS, l = threadIdx.x;
  if (r0 >= m) return;
  const DcArea ar = dc_area(c, b);
  const int K = (m + DC_BLOCK - 1) / DC_BLOCK;
  for (int r = 0; r < DG_ROWS; ++r)
    s_az[r][l] = r0 + r < m ? ar.AZ[(size_t)(r0 + r) * DC_K + l] : 0.f;
  __syncthreads();
  float acc[DG_ROWS];
#pragma unroll
  for (int r = 0; r < DG_ROWS; ++r) acc[r] = 0.f;
  for (int k = 0; k < K; k += 4) {  // (entries beyond K are zero)
    float a[4];
#pragma unroll
    for (int e = 0; e < 4; ++e) a[e] = ar.Ai[(k + e) * DC_K + l];
#pragma unroll
    for (int r = 0; r < DG_ROWS; ++r) {
      const float4 z = *reinterpret_cast<const float4 *>(&s_az[r][k]);
      acc[r] = fmaf(z.x, a[0], fmaf(z.y, a[1], fmaf(z.z, a[2], fmaf(z.w, a[3], acc[r]))));
    }
  }
#pragma unroll
  for (int r = 0; r < DG_ROWS; ++r)
    if (r0 + r < m) ar.G[(size_t)(r0 + r) * DC_K + l] = acc[r];
}

// Barrier counters and start sums of the solves, a CTA per structure.
__global__ void __launch_bounds__(256) dcg_clear_kernel(Ctx c) {
  const DcArea ar = dc_area(c, blockIdx.x);
  for (int k = threadIdx.x; k < EEQ_BIG_REFINE * 2 * DC_K; k += 256) ar.tr[k] = 0.f;
  if (threadIdx.x < EEQ_BIG_REFINE) ar.counter[threadIdx.x] = 0u;
}

// V <- FP32 solution of A d = V (NR right-hand sides) of every structure whose
// refinement (iteration ``it``) is not done.
template <int NR, bool VEC>
__global__ void __launch_bounds__(DC_THREADS, 1) eeq_dcg_kernel(Ctx c, int it) {
  extern __shared__ __align__(16) unsigned char s_raw[];
  DcSmem &sm = *reinterpret_cast<DcSmem *>(s_raw);
  const int N = c.N, ranks = gridDim.x, rank = blockIdx.x;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int i = tid >> 2, q = tid & 3;  // row of the slice, quarter of a G row / right-hand side
  if (group_gave_up(c.w.status)) return;
  if (tid == 0) sm.dead = 0;
  for (int b = 0; b < c.B; ++b) {
    const int m = c.w.n_real[b];
    if (m == 0 || dc_skip(c, b, it, NR)) continue;
    const DcArea ar = dc_area(c, b);
    const float *Hi = c.w.eeq_hi + (size_t)b * N * N;
    float *V = c.w.eeq_V + (size_t)b * 2 * N;
    unsigned *counter = ar.counter + it;
    unsigned passed = 0;
    const int K = (m + DC_BLOCK - 1) / DC_BLOCK, NB = (m + DC_TILE - 1) / DC_TILE;
    const long long tiles = (long long)NB * (NB + 1) / 2;
    const int t0 = (int)(tiles * rank / ranks), t1 = (int)(tiles * (rank + 1) / ranks);
    const int k0 = (int)((long long)rank * m / ranks);
    const int k1 = (int)((long long)(rank + 1) * m / ranks);
    const int len = k1 - k0, row = k0 + i;
    const bool rok = i < len, own = rok && q < NR;
    const size_t o = own ? q * dc_pad(N) + row : 0, oV = own ? (size_t)q * N + row : 0;
    __syncthreads();  // the last structure's shared memory is free
    for (int e = tid; e < len * (DC_K / 4); e += DC_THREADS) {
      const int r = e / (DC_K / 4), k = 4 * (e % (DC_K / 4));
      *reinterpret_cast<float4 *>(&sm.G[r * DC_LDG + k]) =
          *reinterpret_cast<const float4 *>(&ar.G[(size_t)(k0 + r) * DC_K + k]);
    }
    float top = 0.f;
    for (int k = warp; k < DC_K; k += DC_WARPS) {  // Z^T b
      const int l = DC_BLOCK * k + lane;
#pragma unroll
      for (int p = 0; p < NR; ++p) {
        const float *Vp = V + (size_t)p * N;
        const float v0 = l < m ? __ldcg(Vp + l) : 0.f;
        const float v1 = l + 32 < m ? __ldcg(Vp + l + 32) : 0.f;
        top = fmaxf(top, fmaxf(fabsf(v0), fabsf(v1)));
        const float s = warp_sumf(v0 + v1);
        if (lane == 0) sm.tb[p][k] = s;
      }
    }
    // The solve runs on b times a power of two: no product of two residuals leaves
    // FP32's range then, whatever the energies' weights.
    top = warp_maxf(top);
    if (lane == 0) sm.red[warp][0] = top;
    __syncthreads();
#pragma unroll
    for (int w = 0; w < DC_WARPS; ++w) top = fmaxf(top, sm.red[w][0]);
    const float sc = scale_to_one(top);
    if (NR == 1 && it == 0 && rank == 0 && tid == 0) *ar.top = top;
    for (int k = tid; k < NR * DC_K; k += DC_THREADS) sm.tb[k / DC_K][k % DC_K] *= sc;
    // G t of the thread's row and right-hand side: four lanes share a row
    auto project = [&](const float (&tv)[2][DC_K]) {
      float s[NR];
#pragma unroll
      for (int p = 0; p < NR; ++p) s[p] = 0.f;
      if (rok) {
        const float *g = &sm.G[i * DC_LDG];
        for (int k = 4 * q; k < K; k += 16) {
          const float4 gv = *reinterpret_cast<const float4 *>(g + k);
#pragma unroll
          for (int p = 0; p < NR; ++p) {
            const float4 t4 = *reinterpret_cast<const float4 *>(&tv[p][k]);
            s[p] = fmaf(gv.x, t4.x, fmaf(gv.y, t4.y, fmaf(gv.z, t4.z, fmaf(gv.w, t4.w, s[p]))));
          }
        }
      }
#pragma unroll
      for (int p = 0; p < NR; ++p) {
        s[p] += __shfl_xor_sync(0xffffffffu, s[p], 1);
        s[p] += __shfl_xor_sync(0xffffffffu, s[p], 2);
      }
      return NR == 2 && q == 1 ? s[NR - 1] : s[0];
    };
    // mu += G^T u of the slice: a column per thread (NR = 1: two threads each)
    auto restrict_u = [&](float u, float *mu) {
      if (own) sm.x[q][i] = u;
      __syncthreads();
      const int e = tid / DC_K, k = tid % DC_K;
      if (k < K) {
        float a = 0.f;
#pragma unroll 4
        for (int l = NR == 1 ? e : 0; l < len; l += NR == 1 ? 2 : 1)
          a = fmaf(sm.G[l * DC_LDG + k], sm.x[NR == 1 ? 0 : e][l], a);
        atomicAdd(mu + (rank % DC_COPIES * 2 + (NR == 1 ? 0 : e)) * DC_K + k, a);
      }
    };
    // partial (r, u) and max |r| (and (b, b / diag)) of the slice; sums over ranks
    auto publish = [&](float ru, float mx, float bb) {
      float v[3 * NR];
#pragma unroll
      for (int p = 0; p < NR; ++p) {
        const bool mine = own && q == p;
        v[p] = mine ? ru : 0.f;
        v[NR + p] = mine ? bb : 0.f;
        v[2 * NR + p] = mine ? mx : 0.f;
      }
      dc_cta_sum<3 * NR, 2 * NR>(v, sm);
      if (tid == 0)
#pragma unroll
        for (int p = 0; p < NR; ++p)
          __stcg(&ar.norm[2 * rank + p], make_float4(v[p], v[2 * NR + p], v[NR + p], 0.f));
    };
    // (one warp per CTA and right-hand side: the CTAs all read the same lines)
    auto norms = [&](float (&g)[NR], float (&mx)[NR], float (&bb)[NR]) {
      if (warp < NR) {
        float a = 0.f, x = 0.f, d = 0.f;
#pragma unroll 5
        for (int k = lane; k < ranks; k += 32) {
          const float4 v = __ldcg(&ar.norm[2 * k + warp]);
          a += v.x;
          x = fmaxf(x, v.y);
          d += v.z;
        }
        a = warp_sumf(a);
        x = warp_maxf(x);
        d = warp_sumf(d);
        if (lane == 0) sm.sum[warp] = make_float4(a, x, d, 0.f);
      }
      __syncthreads();
#pragma unroll
      for (int p = 0; p < NR; ++p) {
        g[p] = sm.sum[p].x;
        mx[p] = sm.sum[p].y;
        bb[p] = sm.sum[p].z;
      }
    };
    __syncthreads();
    const float bv = own ? __ldcg(V + oV) * sc : 0.f;
    const float dinv = own ? 1.0f / __ldg(Hi + (size_t)row * N + row) : 0.f;
    float r = bv - project(sm.tb), p = 0.f, s = 0.f, x = 0.f;
    if (!own) r = 0.f;
    if (own) {
      atomicAdd(ar.tr + (2 * it + q) * DC_K + row / DC_BLOCK, r);
      __stcg(ar.w[0] + o, 0.f);
      __stcg(ar.w[1] + o, 0.f);
    }
    if (rank < DC_COPIES)
      for (int k = tid; k < 2 * DC_K; k += DC_THREADS) {
        __stcg(ar.mu[0] + rank * 2 * DC_K + k, 0.f);
        __stcg(ar.mu[1] + rank * 2 * DC_K + k, 0.f);
      }
    if (rank == 0)
      for (int k = tid; k < NR * DC_K; k += DC_THREADS) {
        __stcg(ar.t[0] + k, 0.f);
        __stcg(ar.t[1] + k, 0.f);
      }
    if (!group_barrier(counter, (unsigned)ranks * ++passed, sm.dead, c.w.status)) return;
    // what FP32 left in the deflated modes, once more
    for (int k = tid; k < NR * DC_K; k += DC_THREADS) {
      const float t = __ldcg(ar.tr + 2 * it * DC_K + k);
      sm.t[k / DC_K][k % DC_K] = t;
      sm.tb[k / DC_K][k % DC_K] += t;
    }
    __syncthreads();
    r -= project(sm.t);
    if (!own) r = 0.f;
    float u = dinv * r;
    if (own) __stcg(ar.u + o, u);
    restrict_u(u, ar.mu[1]);
    if (rank == 1 % ranks)
      for (int k = m + tid; k < DC_TILE * NB; k += DC_THREADS)
#pragma unroll
        for (int e = 0; e < NR; ++e) __stcg(ar.u + e * dc_pad(N) + k, 0.f);
    publish(r * u, fabsf(r), bv * dinv * bv);
    if (!group_barrier(counter, (unsigned)ranks * ++passed, sm.dead, c.w.status)) return;
    float g[NR], g0[NR], mx[NR], bb[NR], stop[NR], alpha[NR], beta[NR];
    bool on[NR], more = false;
    norms(g, mx, bb);
    const float end = it == 0 ? 0.f : dc_bars(c, b, NR).end * sc;
#pragma unroll
    for (int e = 0; e < NR; ++e) {
      g0[e] = g[e];
      stop[e] = fmaxf(DC_GAIN * g[e], DC_FLOOR * bb[e]);
      on[e] = g[e] > stop[e] && mx[e] > end;
      more |= on[e];
      alpha[e] = beta[e] = 0.f;
    }
    int par = 0;
    for (int n = 0; n < DC_ITS && more; ++n) {
      // u in the complement: A (u - Z mu) = P A u
      for (int k = tid; k < NR * DC_K; k += DC_THREADS) {
        float a = 0.f;
#pragma unroll
        for (int e = 0; e < DC_COPIES; ++e) a += __ldcg(ar.mu[par ^ 1] + e * 2 * DC_K + k);
        sm.mu[k / DC_K][k % DC_K] = a;
      }
      __syncthreads();
      if (own) u -= sm.mu[q][row / DC_BLOCK];
      dc_product<NR, VEC>(Hi, N, m, t0, t1, ar.u, ar.w[par], ar.t[par], sm);
      if (!group_barrier(counter, (unsigned)ranks * ++passed, sm.dead, c.w.status)) return;
      float v = own ? __ldcg(ar.w[par] + o) : 0.f;
      for (int k = tid; k < NR * DC_K; k += DC_THREADS) {
        sm.t[k / DC_K][k % DC_K] = __ldcg(ar.t[par] + k);
        if (rank < DC_COPIES && n > 0) __stcg(ar.mu[par] + rank * 2 * DC_K + k, 0.f);
        if (rank == 0 && n > 0) __stcg(ar.t[par ^ 1] + k, 0.f);
      }
      if (own && n > 0) __stcg(ar.w[par ^ 1] + o, 0.f);
      __syncthreads();
      v -= project(sm.t);
      {
        // (r, u - Z mu), not (r, u): r keeps a rounding error in the deflated modes
        float d[2 * NR];
#pragma unroll
        for (int e = 0; e < NR; ++e) {
          d[2 * e] = own && q == e ? v * u : 0.f;
          d[2 * e + 1] = own && q == e ? r * u : 0.f;
        }
        dc_cta_sum<2 * NR, 2 * NR>(d, sm);
        if (tid == 0)
#pragma unroll
          for (int e = 0; e < NR; ++e)
            __stcg(ar.dot + 2 * rank + e, make_float2(d[2 * e], d[2 * e + 1]));
      }
      if (!group_barrier(counter, (unsigned)ranks * ++passed, sm.dead, c.w.status)) return;
      if (warp < NR) {
        float d = 0.f, ru = 0.f;
#pragma unroll 5
        for (int k = lane; k < ranks; k += 32) {
          const float2 t = __ldcg(ar.dot + 2 * k + warp);
          d += t.x;
          ru += t.y;
        }
        d = warp_sumf(d);
        ru = warp_sumf(ru);
        if (lane == 0) sm.dot[warp] = make_float2(d, ru);
      }
      __syncthreads();
      bool bad = false, definite = true;
#pragma unroll
      for (int e = 0; e < NR; ++e) {
        const float d = sm.dot[e].x, ru = sm.dot[e].y;
        if (!on[e]) {
          alpha[e] = beta[e] = 0.f;
          continue;
        }
        beta[e] = n == 0 ? 0.f : ru / g[e];
        g[e] = ru;
        const float den = n == 0 ? d : d - beta[e] * ru / alpha[e];
        if (!(den > 0.f)) {  // (p, P A p): as in d4_eeq_cg.cu
          bad = true;
          definite = definite && n > 0 && d > 0.f && ru <= DC_LAST * g0[e];
        }
        alpha[e] = ru / den;
      }
      if (bad) {
        if (!definite && tid == 0) set_status(c.w.status, D4_ERR_EEQ_SINGULAR);
        break;
      }
      const float al = NR == 2 && q == 1 ? alpha[NR - 1] : alpha[0];
      const float be = NR == 2 && q == 1 ? beta[NR - 1] : beta[0];
      if (own) {
        p = fmaf(be, p, u);
        s = fmaf(be, s, v);
        x = fmaf(al, p, x);
        r = fmaf(-al, s, r);
        u = dinv * r;
        __stcg(ar.u + o, u);
      }
      restrict_u(u, ar.mu[par]);
      publish(r * u, fabsf(r), 0.f);
      par ^= 1;
      if (!group_barrier(counter, (unsigned)ranks * ++passed, sm.dead, c.w.status)) return;
      float gn[NR];
      norms(gn, mx, bb);
      more = false;
#pragma unroll
      for (int e = 0; e < NR; ++e) {
        on[e] = on[e] && gn[e] > stop[e] && mx[e] > end;
        more |= on[e];
      }
    }
    // d = x + Z (Z^T A Z)^-1 Z^T b
    const int kb = k0 / DC_BLOCK;  // the slice's blocks: three at most
    if (warp < 4 * NR) {
      const int e = warp >> 2, k = kb + (warp & 3);
      float a = 0.f;
      if (k < K) {
        for (int l = lane; l < K; l += 32) a = fmaf(__ldg(ar.Ai + k * DC_K + l), sm.tb[e][l], a);
        a = warp_sumf(a);
      }
      if (lane == 0) sm.y[e][warp & 3] = a;
    }
    __syncthreads();
    if (own) V[oV] = (x + sm.y[q][row / DC_BLOCK - kb]) / sc;
  }
}

// x += v in double-float; clears the sums of the residual (FP64, in the room of
// the products w).
__global__ void __launch_bounds__(256) dcg_update_kernel(Ctx c, int it, int nr) {
  const int b = blockIdx.y, N = c.N, k = blockIdx.x * 256 + threadIdx.x;
  if (k >= c.w.n_real[b] || dc_skip(c, b, it, nr)) return;
  double *sums = reinterpret_cast<double *>(dc_area(c, b).w[0]);
  for (int q = 0; q < nr; ++q) {
    const size_t o = (size_t)b * 2 * N + (size_t)q * N + k;
    const float2 x = c.w.eeq_X[o];
    const dfl s = df_add(dfl{x.x, x.y}, dfl{c.w.eeq_V[o], 0.f});
    c.w.eeq_X[o] = make_float2(s.hi, s.lo);
    sums[q * dc_pad(N) + k] = 0.0;
  }
}

struct DrSmem {
  float2 z[2][2][DC_WARPS][DC_TILE];  // [turn][right-hand side][warp]: a tile's column sums
  float2 xj[2][2][DC_TILE], xi[2][DC_TILE];  // x of a tile's columns, rows
};

// (hi + lo) x in double-float, summed in FP64 at L2, over the stored half of the
// matrix: dc_product's tiles, each for both of its products, with four of a
// warp's eight rows of both planes in flight.  Bound by the latency of its FP32
// sums (12 instructions per entry, product and right-hand side): 16000 atoms, two
// right-hand sides 0.37 ms (2.8 TB/s), one 0.21 ms (4.8 TB/s); five of them 1.5 ms
// against 2.0 over the whole matrix.  256 threads with eight rows in
// flight 0.38 and 0.22, two rows of 16 warps 0.39 and 0.24.
template <int NR, bool VEC>
__global__ void __launch_bounds__(DC_THREADS, 1) dcg_residual_kernel(Ctx c, int it) {
  extern __shared__ __align__(16) unsigned char s_raw[];
  DrSmem &sm = *reinterpret_cast<DrSmem *>(s_raw);
  const int b = blockIdx.y, N = c.N, m = c.w.n_real[b];
  if (m == 0 || dc_skip(c, b, it, NR)) return;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int NB = (m + DC_TILE - 1) / DC_TILE;
  const long long tiles = (long long)NB * (NB + 1) / 2;
  const int t0 = (int)(tiles * blockIdx.x / gridDim.x);
  const int t1 = (int)(tiles * (blockIdx.x + 1) / gridDim.x);
  if (t0 >= t1) return;
  const float *Hi = c.w.eeq_hi + (size_t)b * N * N, *Lo = c.w.eeq_lo + (size_t)b * N * N;
  const float2 *X = c.w.eeq_X + (size_t)b * 2 * N;
  double *sums = reinterpret_cast<double *>(dc_area(c, b).w[0]);
  const size_t us = dc_pad(N);
  constexpr int W = 4;  // rows in flight
  static_assert(DC_ROWS % W == 0 && NR * DC_TILE <= DC_THREADS, "the warp's rows");
  auto col = [&](int J, int e) { return DC_TILE * J + (VEC ? 4 * lane + e : lane + 32 * e); };
  auto load_row = [&](float (&h)[4], float (&g)[4], int I, int J, int r) {  // as in dc_product
    const size_t o = (size_t)min(DC_TILE * I + DC_ROWS * warp + r, m - 1) * N;
    if (VEC) {
      const size_t p = o + min(col(J, 0), N - 4);
      const float4 v = dc_stream4(Hi + p), w = dc_stream4(Lo + p);
      h[0] = v.x, h[1] = v.y, h[2] = v.z, h[3] = v.w;
      g[0] = w.x, g[1] = w.y, g[2] = w.z, g[3] = w.w;
    } else {
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const size_t p = o + min(col(J, e), m - 1);
        h[e] = __ldg(Hi + p), g[e] = __ldg(Lo + p);
      }
    }
  };
  const int xq = tid / DC_TILE, xk = tid % DC_TILE;  // an x entry per thread
  auto load_x = [&](int J) {
    const int k = DC_TILE * J + xk;
    return xq < NR && k < m ? __ldg(X + (size_t)xq * N + k) : make_float2(0.f, 0.f);
  };
  // acc += (h + g) x, the low part unnormalised
  auto add = [](dfl &acc, float h, float g, float2 x) {
    const float p = h * x.x;
    const float e = fmaf(h, x.y, fmaf(g, x.x, fmaf(h, x.x, -p)));
    const dfl s = df_two_sum(acc.hi, p);
    acc = {s.hi, acc.lo + (s.lo + e)};
  };
  int I, J;
  tri_entry(t0, I, J);
  float h[W][4], g[W][4];
  dfl y[DC_ROWS][NR];
#pragma unroll
  for (int r = 0; r < W; ++r) load_row(h[r], g[r], I, J, r);
  if (xq < NR) sm.xj[0][xq][xk] = load_x(J);
  bool first = true;
  int turn = 0;
  for (int t = t0; t < t1; ++t) {
    if (first || J == 0) {  // a new row of tiles
      first = false;
      const float2 xi = load_x(I);
      __syncthreads();
      if (xq < NR) sm.xi[xq][xk] = xi;
      __syncthreads();
#pragma unroll
      for (int r = 0; r < DC_ROWS; ++r)
#pragma unroll
        for (int q = 0; q < NR; ++q) y[r][q] = {0.f, 0.f};
    }
    const bool diag = J == I, more = t + 1 < t1;
    const int In = diag ? I + 1 : I, Jn = diag ? 0 : J + 1;
    const float2 xn = load_x(more ? Jn : J);
    float2 xj[NR][4];
    dfl z[NR][4];
#pragma unroll
    for (int q = 0; q < NR; ++q)
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        xj[q][e] = sm.xj[turn][q][VEC ? 4 * lane + e : lane + 32 * e];
        z[q][e] = {0.f, 0.f};
      }
    const bool edge = DC_TILE * (J + 1) > m;
#pragma unroll
    for (int r = 0; r < DC_ROWS; ++r) {
      float (&hr)[4] = h[r % W], (&gr)[4] = g[r % W];
      if (edge) {
#pragma unroll
        for (int e = 0; e < 4; ++e)
          if (col(J, e) >= m) hr[e] = gr[e] = 0.f;
      }
#pragma unroll
      for (int q = 0; q < NR; ++q) {
        const float2 xi = sm.xi[q][DC_ROWS * warp + r];
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          add(y[r][q], hr[e], gr[e], xj[q][e]);
          add(z[q][e], hr[e], gr[e], xi);
        }
      }
      if (r + W < DC_ROWS) load_row(hr, gr, I, J, r + W);
      else if (more) load_row(hr, gr, In, Jn, r + W - DC_ROWS);
    }
    if (xq < NR) sm.xj[turn ^ 1][xq][xk] = xn;
    if (!diag) {  // the mirrored tile's product, summed over the warps
#pragma unroll
      for (int q = 0; q < NR; ++q)
#pragma unroll
        for (int e = 0; e < 4; ++e)
          sm.z[turn][q][warp][VEC ? 4 * lane + e : lane + 32 * e] =
              make_float2(z[q][e].hi, z[q][e].lo);
      __syncthreads();
      if (xq < NR) {
        dfl s = {0.f, 0.f};
#pragma unroll
        for (int v = 0; v < DC_WARPS; ++v) {
          const float2 a = sm.z[turn][xq][v][xk];
          const dfl n = df_two_sum(s.hi, a.x);
          s = {n.hi, s.lo + (n.lo + a.y)};
        }
        atomicAdd(sums + xq * us + DC_TILE * J + xk, (double)s.hi + (double)s.lo);
      }
    }
    if (diag || !more) {  // the row of tiles ends
#pragma unroll
      for (int r = 0; r < DC_ROWS; ++r)
#pragma unroll
        for (int q = 0; q < NR; ++q) {
          dfl a = y[r][q];
#pragma unroll
          for (int o = 16; o > 0; o >>= 1) {
            const float oh = __shfl_xor_sync(0xffffffffu, a.hi, o);
            const float ol = __shfl_xor_sync(0xffffffffu, a.lo, o);
            const dfl s = df_two_sum(a.hi, oh);
            a = df_fast(s.hi, s.lo + (a.lo + ol));
          }
          const int row = DC_TILE * I + DC_ROWS * warp + r;
          if (lane == 0 && row < m) atomicAdd(sums + q * us + row, (double)a.hi + (double)a.lo);
        }
    }
    turn ^= 1;
    I = In;
    J = Jn;
  }
}

// v <- FP32 r = b - A x and the structure's max |r| of the iteration.
__global__ void __launch_bounds__(256) dcg_rest_kernel(Ctx c, int it, int nr) {
  const int b = blockIdx.y, N = c.N, k = blockIdx.x * 256 + threadIdx.x;
  const int m = c.w.n_real[b];
  if (blockIdx.x * 256 >= m) return;
  if (dc_skip(c, b, it, nr)) {
    if (k == 0) c.w.eeq_res[b * EEQ_BIG_REFINE + it] = c.w.eeq_res[b * EEQ_BIG_REFINE + it - 1];
    return;
  }
  const double *sums = reinterpret_cast<const double *>(dc_area(c, b).w[0]);
  float mx = 0.f;
  if (k < m)
    for (int q = 0; q < nr; ++q) {
      const size_t o = (size_t)b * 2 * N + (size_t)q * N + k;
      const float2 bb = c.w.eeq_B[o];
      const float r = (float)((double)bb.x - sums[q * dc_pad(N) + k] + (double)bb.y);
      c.w.eeq_V[o] = r;
      mx = fmaxf(mx, fabsf(r));
    }
  mx = warp_maxf(mx);
  if ((threadIdx.x & 31) == 0)
    atomicMax(&c.w.eeq_res[b * EEQ_BIG_REFINE + it], __float_as_uint(mx));
}

namespace {

int dc_sms() {
  const int n = sm_count();
  return n < (int)DC_RANKS ? n : (int)DC_RANKS;
}

template <int NR, bool VEC>
bool launch_solve(const Ctx &c, cudaStream_t st, int it) {
  if (c.flags & D4_FLAG_TEST_FALLBACK) return false;
  Ctx cc = c;
  void *args[] = {&cc, &it};
  const void *f = reinterpret_cast<const void *>(&eeq_dcg_kernel<NR, VEC>);
  ensure_smem_impl(f, sizeof(DcSmem));
  keep_error();  // (a refused launch of this kernel itself is no error of the call)
  if (cudaLaunchCooperativeKernel(f, dim3((unsigned)dc_sms()), dim3(DC_THREADS), args,
                                  sizeof(DcSmem), st) != cudaSuccess) {
    cudaGetLastError();
    return false;
  }
  return true;
}

template <int NR, bool VEC>
void launch_residual(const Ctx &c, cudaStream_t st, int it) {
  const dim3 rows((c.N + 255) / 256, c.B);
  dcg_update_kernel<<<rows, 256, 0, st>>>(c, it, NR);
  ensure_smem(dcg_residual_kernel<NR, VEC>, (int)sizeof(DrSmem));
  dcg_residual_kernel<NR, VEC><<<dim3(dc_sms(), c.B), DC_THREADS, sizeof(DrSmem), st>>>(c, it);
  dcg_rest_kernel<<<rows, 256, 0, st>>>(c, it, NR);
}

}  // namespace

// Whether deflated conjugate gradients solve the batch: one or two structures
// in spatial order whose matrices outgrow L2.  Charges + adjoint in us, against
// plain conjugate gradients (d4_eeq_cg.cu) 1 x 4000 atoms 2129 / 1822, 1 x 4500
// 2249 / 2019 and 1 x 5000 2378 / 4419; against the factorisation 1 x 6001 3042 /
// 5645, 1 x 16000 12087 / 22010, 2 x 4000 3768 / 3983, 2 x 6001 5696 / 6729, but 3 x
// 5000 6462 / 5845 and 4 x 5000 8473 / 6456 (structures run one after the other
// here).
bool eeq_dcg_takes(const Ctx &c) {
  if (!c.zsorted || c.B > 2 || c.N > DC_K * DC_BLOCK) return false;
  if ((size_t)4 * c.B * c.N * c.N <= (size_t)84 << 20) return false;
  const int sms = dc_sms();
  if (sms < DC_COPIES || (c.N + sms - 1) / sms > DC_SLICE) return false;
  return 4 * dc_floats(c.N) <= dc_stride(c.N);
}

bool launch_eeq_dcg(const Ctx &c, cudaStream_t st, bool adjoint) {
  const int B = c.B, N = c.N;
  if (!adjoint) {
    const unsigned nk = (N + DC_BLOCK - 1) / DC_BLOCK;
    dcg_az_kernel<<<dim3(nk * (nk + 1) / 2, B), 256, 0, st>>>(c);
    dcg_a0_kernel<<<dim3(nk, B), DC_K, 0, st>>>(c);
    dcg_inverse_kernel<<<B, 1024, 0, st>>>(c);
    dcg_g_kernel<<<dim3((N + DG_ROWS - 1) / DG_ROWS, B), DC_K, 0, st>>>(c);
  }
  dcg_clear_kernel<<<B, 256, 0, st>>>(c);
  launch_eeq_big_rhs(c, st, adjoint);
  const bool vec = N % 4 == 0;
  for (int it = 0; it < EEQ_BIG_REFINE; ++it) {
    auto solve = adjoint ? (vec ? &launch_solve<1, true> : &launch_solve<1, false>)
                         : (vec ? &launch_solve<2, true> : &launch_solve<2, false>);
    if (!solve(c, st, it)) return false;
    auto residual = adjoint ? (vec ? &launch_residual<1, true> : &launch_residual<1, false>)
                            : (vec ? &launch_residual<2, true> : &launch_residual<2, false>);
    residual(c, st, it);
  }
  launch_eeq_big_finish(c, st, adjoint, true);
  return true;
}

}  // namespace d4
