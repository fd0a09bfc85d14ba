// FP64 EEQ solve of the plain method: Coulomb matrix, blocked Cholesky
// factorisation, solves of A^-1 b and A^-1 1 with the total-charge
// constraint, and the adjoint solve.
//
// GB300 issues a warp instruction on the FP64 pipe every 64 cycles and SM
// sub-partition, dependent or not, so a single warp gets a quarter of the SM's
// two FMAs per cycle: one SM needs 0.3 ms for the n^3 / 6 FMAs of 200 atoms,
// as much again for the erf terms of their matrix, and anything one warp does
// alone takes four times as long.  The matrix is therefore built by a kernel
// over all rows of the batch, structures padded beyond EEQ64_SMALL atoms are
// factorised panel by panel (32 columns) by all SMs, two launches per panel,
// and smaller ones stay in one CTA's shared memory, one launch.  Both run the
// same steps.  A panel: one warp forms the pivots on a sub-partition of its
// own (a chain of ~500 cycles per column), the others update the 32 x 32
// diagonal block and carry the rows below it, one column behind.  The trailing
// matrix: a warp per 32 rows (a lane each) and a few columns.  The right-hand
// sides ride along as two more rows of the matrix, which makes their forward
// substitution part of the factorisation, and the rows of the identity give
// the inverse of each diagonal block, which the triangular solves use.
//
// Measured (EEQ stage / adjoint): 64 structures of 8..200 atoms 1757 / 454 ->
// 480 / 45 us, 301 atoms 8623 / 766 -> 385 / 78 us, 57 atoms 245 / 98 ->
// 78 / 14 us, 32 atoms 122 -> 42 us; before, one CTA per structure
// eliminated column by column (three barriers each) and one warp solved row
// by row.
#include "d4_common.cuh"
#include "d4_fpmath.cuh"
#include "d4_kernels.cuh"

namespace d4 {

namespace {

constexpr int EB = 32;            // panel width
constexpr int EEQ64_SMALL = 96;   // one-CTA path up to this padded size (three panels: ~7 us
                                  // of launches saved; beyond, one SM's n^3 / 6 dominates)
constexpr unsigned FULL = 0xffffffffu;

__device__ __forceinline__ int eeq64_order(const Ctx &c, int b) {  // real atoms
  const int n = c.w.n_eff[b];
  return n > 0 ? c.w.cidx[(size_t)b * c.N + n - 1] + 1 : 0;
}
__device__ __forceinline__ double *eeq64_factor(const Ctx &c, int b) {
  return c.w.eeq_L + (size_t)b * ((size_t)c.N * (c.N + 1) / 2);
}
// Inverses of the diagonal blocks until the factor takes them (32 x 32 each,
// row-major), in the room of the pair records, which are written later.
__device__ __forceinline__ double *eeq64_inv(const Ctx &c, int b) {
  return c.w.pr_r + (size_t)b * ((c.N + EB - 1) / EB) * EB * EB;
}
// Row r of the right-hand sides, compact order (b, then 1), in the room of
// arrays the adjoint writes later.
__device__ __forceinline__ double *eeq64_rhs(const Ctx &c, int b, int r) {
  return (r == 0 ? c.w.eeq_w : c.w.dEdq) + (size_t)b * c.N;
}

// Where the rows that pass through a panel live.  Row w of the panel at k0:
// w < 32 row w of the identity (its result is column w of the inverse X of
// the diagonal block), then the matrix rows below the block, then the two
// right-hand sides.
struct PanelRows {
  double *L, *X;        // X: 32 x 32 row-major, or nullptr for the block's own packed place
  double *v0, *v1;
  int k0, kb, m;
  __device__ __forceinline__ int count() const { return EB + (m - k0 - kb) + 2; }
  __device__ __forceinline__ double load(int w, int j) const {
    if (w < EB) return j == w ? 1.0 : 0.0;
    const int i = k0 + kb + w - EB;
    if (i < m) return L[tri_index(i, k0 + j)];  // rows below the block: kb = 32
    return (i < m + 2 && j < kb) ? (i == m ? v0 : v1)[k0 + j] : 0.0;
  }
  __device__ __forceinline__ void store(int w, int j, double x) const {
    if (w < EB) {
      if (X)
        X[j * EB + w] = x;
      else if (j < kb && w <= j)
        L[tri_index(k0 + j, k0 + w)] = x;
      return;
    }
    const int i = k0 + kb + w - EB;
    if (i < m)
      L[tri_index(i, k0 + j)] = x;
    else if (i < m + 2 && j < kb)
      (i == m ? v0 : v1)[k0 + j] = x;
  }
};

struct PanelSmem {
  double L[EB * EB];   // [c][r]: column c of the factor
  double inv[EB];      // 1 / pivot
  double next[2][EB];  // the column after the next, all but its last update applied
  double o[2][4][EB];  // the rows' scaled entries of the last two columns
};

// Pivot of column c, whose entries (a lane per row) are `a`: the scaled column
// and 1 / sqrt(d) to shared memory.
__device__ __forceinline__ void eeq64_pivot(double a, int c, PanelSmem &sm, int *status) {
  const int lane = threadIdx.x & 31;
  double d = __shfl_sync(FULL, a, c);
  // d > 0 by its high word (a comparison would take the FP64 pipe)
  const int hi = __double2hiint(d);
  if (hi <= 0 || hi > 0x7ff00000) {
    if (lane == 0) set_status(status, D4_ERR_EEQ_SINGULAR);
    d = 1.0;
  }
  if (lane == c) a = d;
  const double inv = rsqrt_pos<false>(d);  // (finite: a matrix with an infinite entry has NaN)
  sm.L[c * EB + lane] = lane >= c ? a * inv : 0.0;
  if (lane == c) sm.inv[c] = inv;
}

// The panel of R by the CTA's eight warps.  Warp 0 forms the pivots: it takes
// the next column from shared memory, applies its last update and scales it.
// Warps 1-3 hold the diagonal block (lane = row, columns 3 t + g; rows beyond
// the matrix are the identity), warps 5-7 carry the rows w0 .. w0 + 32 S - 1
// through it (lane = row, the same columns), one column behind.  Warp w runs
// on sub-partition w % 4, so the pivots (seven dependent FP64 instructions
// per column) have a pipe of their own; one barrier per column.
template <int S>
__device__ __forceinline__ void eeq64_panel(const PanelRows &R, int w0, PanelSmem &sm,
                                            int *status) {
  constexpr int NC = (EB + 2) / 3;  // columns per warp
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = (warp & 3) - 1;
  const bool pivot = warp == 0, diag = warp < 4 && g >= 0, rows = warp >= 4 && g >= 0;
  double x[S][NC];
  if (pivot || diag) {
    const double *row = R.L + tri_index(R.k0 + (lane < R.kb ? lane : 0), R.k0);
    auto entry = [&](int j) {
      return (lane < R.kb && j <= lane) ? row[j] : (j == lane ? 1.0 : 0.0);
    };
    if (pivot) {
      const double c1 = entry(1);
      eeq64_pivot(entry(0), 0, sm, status);
      sm.next[1][lane] = c1;
    } else {
#pragma unroll
      for (int t = 0; t < NC; ++t) x[0][t] = 3 * t + g < EB ? entry(3 * t + g) : 0.0;
    }
  } else if (rows) {
#pragma unroll
    for (int s = 0; s < S; ++s)
#pragma unroll
      for (int t = 0; t < NC; ++t)
        x[s][t] = 3 * t + g < EB ? R.load(w0 + 32 * s + lane, 3 * t + g) : 0.0;
  }
#pragma unroll
  for (int c = 0; c < EB; ++c) {
    __syncthreads();
    if (pivot) {
      if (c + 1 < EB) {
        const double *col = sm.L + c * EB;
        eeq64_pivot(fma(-col[lane], col[c + 1], sm.next[(c + 1) & 1][lane]), c + 1, sm, status);
      }
    } else if (diag) {
      if (c + 2 < EB) {  // columns c + 2 .. 31; column c + 2 goes to the pivot warp
        const double *col = sm.L + c * EB;
        const double l = col[lane];
        const int n2 = (c + 2) / 3, g2 = (c + 2) % 3;
        // (entries above the diagonal collect values that are never read)
        if (g >= g2) x[0][n2] = fma(-l, col[min(3 * n2 + g, EB - 1)], x[0][n2]);
        if (g == g2) sm.next[c & 1][lane] = x[0][n2];
#pragma unroll
        for (int t = n2 + 1; t < NC; ++t)
          if (3 * t + 2 < EB || 3 * t + g < EB)
            x[0][t] = fma(-l, col[3 * t + g], x[0][t]);
      }
    } else if (rows) {
      const int n1 = c / 3, g1 = c % 3;
      if (c > 0) {
        const double *col = sm.L + (c - 1) * EB;
#pragma unroll
        for (int s = 0; s < S; ++s) {
          const double o = -sm.o[(c - 1) & 1][s][lane];
          if (g >= g1) x[s][n1] = fma(o, col[min(3 * n1 + g, EB - 1)], x[s][n1]);
#pragma unroll
          for (int t = n1 + 1; t < NC; ++t)
            if (3 * t + 2 < EB || 3 * t + g < EB) x[s][t] = fma(o, col[3 * t + g], x[s][t]);
        }
      }
      if (g == g1) {
        const double inv = sm.inv[c];
#pragma unroll
        for (int s = 0; s < S; ++s) {
          x[s][n1] *= inv;
          sm.o[c & 1][s][lane] = x[s][n1];
        }
      }
    }
  }
  if (rows) {
    const int n = R.count();
#pragma unroll
    for (int s = 0; s < S; ++s) {
      const int w = w0 + 32 * s + lane;
      if (w < n) {
#pragma unroll
        for (int t = 0; t < NC; ++t)
          if (3 * t + g < EB) R.store(w, 3 * t + g, x[s][t]);
      }
    }
  }
}

// Trailing update of tile (ti, tj, part): rows t0 + 32 ti .. (a lane each),
// the CW columns t0 + 32 tj + CW part ..; sj: the columns' panel rows, [32][CW],
// or nullptr to read them from L.  The first columns' tiles also take the
// right-hand sides.
template <int CW>
__device__ __forceinline__ void eeq64_update_tile(double *L, const double *sj, double *v0,
                                                  double *v1, int ti, int tj, int part, int k0,
                                                  int t0, int m) {
  const int lane = threadIdx.x & 31;
  const int i = t0 + 32 * ti + lane, j0 = t0 + 32 * tj + CW * part;
  if (j0 >= m || j0 > t0 + 32 * ti + 31) return;  // beyond the matrix or above the diagonal
  const bool live = i < m;
  const double *row = L + tri_index(live ? i : m - 1, k0);
  const bool rhs = tj == 0 && part == 0;
  double acc[CW], r0 = 0.0, r1 = 0.0;
#pragma unroll
  for (int q = 0; q < CW; ++q) acc[q] = 0.0;
#pragma unroll 8
  for (int cc = 0; cc < EB; ++cc) {
    const double x = row[cc];
#pragma unroll
    for (int q = 0; q < CW; ++q)
      acc[q] = fma(x, sj ? sj[cc * CW + q] : L[tri_index(min(j0 + q, m - 1), k0 + cc)], acc[q]);
  }
  if (rhs) {
#pragma unroll 8
    for (int cc = 0; cc < EB; ++cc) {
      const double x = row[cc];
      r0 = fma(x, v0[k0 + cc], r0);
      r1 = fma(x, v1[k0 + cc], r1);
    }
  }
  if (live) {
    double *out = L + tri_index(i, 0);
#pragma unroll
    for (int q = 0; q < CW; ++q)
      if (j0 + q <= i) out[j0 + q] -= acc[q];
    if (rhs) {
      v0[i] -= r0;
      v1[i] -= r1;
    }
  }
}

// Block inverse X of block kk: from the packed factor or the scratch of the
// panel kernel.
struct InvAt {
  const double *L, *X;
  __device__ __forceinline__ double at(int k0, int r, int c) const {
    return X ? X[(size_t)k0 * EB + r * EB + c] : L[tri_index(k0 + r, k0 + c)];
  }
};

constexpr int ES_THREADS = 256;
struct SolveSmem {
  double part[4][EB];
  double half[ES_THREADS / 2];
};

// L z = v (FWD) or L^T x = z in place, by the whole CTA of 256 threads.  Per
// block of 32: the product with the block inverse (four warps, eight terms
// each, then their sum), and the other rows (columns), each by two threads
// that take half of the 32 terms; their factor entries are on their way while
// the product runs.
template <bool FWD>
__device__ void eeq64_solve(const double *L, const InvAt &inv, double *v, int m, SolveSmem &sm) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int half = threadIdx.x >> 7, i_off = threadIdx.x & 127;
  constexpr int HB = EB / 2;
  const int nb = (m + EB - 1) / EB;
  for (int blk = 0; blk < nb; ++blk) {
    const int k0 = EB * (FWD ? blk : nb - 1 - blk);
    const int kb = min(EB, m - k0);
    const int first = FWD ? k0 + EB : 0, last = FWD ? m : k0;
    double l[HB];
    auto entries = [&](int i) {
#pragma unroll
      for (int cc = 0; cc < HB; ++cc) {
        const int e = HB * half + cc;
        l[cc] = FWD ? L[tri_index(i, k0 + e)] : (e < kb ? L[tri_index(k0 + e, i)] : 0.0);
      }
    };
    if (first + i_off < last) entries(first + i_off);  // FWD: then kb = 32
    if (warp < 4) {
      double z = 0.0;
#pragma unroll
      for (int cc = 0; cc < 8; ++cc) {
        const int e = 8 * warp + cc;
        const bool ok = lane < kb && e < kb && (FWD ? e <= lane : e >= lane);
        z = fma(ok ? (FWD ? inv.at(k0, lane, e) : inv.at(k0, e, lane)) : 0.0,
                e < kb ? v[k0 + e] : 0.0, z);
      }
      sm.part[warp][lane] = z;
    }
    __syncthreads();
    if (warp == 0 && lane < kb)
      v[k0 + lane] = (sm.part[0][lane] + sm.part[1][lane]) +
                     (sm.part[2][lane] + sm.part[3][lane]);
    __syncthreads();
    for (int i0 = first; i0 < last; i0 += ES_THREADS / 2) {  // block-uniform
      const int i = i0 + i_off;
      double a0 = 0.0, a1 = 0.0;
      if (i < last) {
        const double *xv = v + k0 + HB * half;
#pragma unroll
        for (int cc = 0; cc < HB; cc += 2) {
          const int e = HB * half + cc;
          a0 = fma(l[cc], e < kb ? xv[cc] : 0.0, a0);
          a1 = fma(l[cc + 1], e + 1 < kb ? xv[cc + 1] : 0.0, a1);
        }
        if (i + ES_THREADS / 2 < last) entries(i + ES_THREADS / 2);
        if (half) sm.half[i_off] = a0 + a1;
      }
      __syncthreads();
      if (!half && i < last) v[i] -= (a0 + a1) + sm.half[i_off];
      __syncthreads();
    }
  }
}

// x . y over m entries by the whole CTA (all threads get it).
__device__ double eeq64_dot(const double *x, const double *y, int m, SolveSmem &sm) {
  double s = 0.0;
  for (int k = threadIdx.x; k < m; k += ES_THREADS) s = fma(x[k], y[k], s);
  s = warp_sum(s);
  __syncthreads();
  if ((threadIdx.x & 31) == 0) sm.half[threadIdx.x >> 5] = s;
  __syncthreads();
  s = 0.0;
#pragma unroll
  for (int w = 0; w < ES_THREADS / 32; ++w) s += sm.half[w];
  __syncthreads();
  return s;
}

// Charges from the forward solutions z_b = L^-1 b (v) and z_1 = L^-1 1 (v + ldv):
// 1^T A^-1 b = z_1 . z_b and 1^T A^-1 1 = z_1 . z_1, so the constraint's
// multiplier is known before the backward solve and
// q = A^-1 (b - lambda 1) = L^-T (z_b - lambda z_1) takes one right-hand side.
// By the whole CTA; z_1 stays for the adjoint (eeq_y, compact order).
__device__ void eeq64_charges(const Ctx &c, int b, const double *L, const InvAt &inv, double *v,
                              ptrdiff_t ldv, int m, SolveSmem &sm) {
  const double sx = eeq64_dot(v, v + ldv, m, sm), sy = eeq64_dot(v + ldv, v + ldv, m, sm);
  const double lam = m > 0 ? (sx - c.charge[b]) / sy : 0.0;
  if (threadIdx.x == 0) {
    c.w.eeq_sum[2 * b] = sy;
    c.w.eeq_sum[2 * b + 1] = lam;
  }
  for (int k = threadIdx.x; k < m; k += ES_THREADS) {
    c.w.eeq_y[(size_t)b * c.N + k] = v[ldv + k];
    v[k] = fma(-lam, v[ldv + k], v[k]);
  }
  __syncthreads();
  eeq64_solve<false>(L, inv, v, m, sm);
  for (int i = threadIdx.x; i < c.N; i += ES_THREADS) {
    const size_t a = (size_t)b * c.N + i;
    const int k = c.w.cidx[a];
    c.w.q[a] = k >= 0 ? v[k] : 0.0;
  }
}

}  // namespace

namespace {

constexpr int CS_ATOMS = 16;  // atoms of a group of four warps

// Coordination numbers (D4; EEQ, not capped yet) from the pairs' terms (cn_kernel),
// always in the same order: 16 atoms from ``first`` on per group of four warps (of
// GROUPS in the CTA), two lanes per atom and warp, every eighth partner each, then
// the sums of lanes and warps.  (A lane per partner and sums across all lanes take
// four times the FP64 instructions for small structures.)
template <int GROUPS>
__device__ __forceinline__ void cn64_sum(const Ctx &c, int b, int first) {
  __shared__ double2 s_part[GROUPS][4][CS_ATOMS];
  const int N = c.N, n = c.w.n_eff[b];
  const int group = threadIdx.x >> 7, warp = (threadIdx.x >> 5) & 3, lane = threadIdx.x & 31;
  const int a = first + CS_ATOMS * group + (lane & 15);
  const double2 *M = cn64_terms(c, b);
  double2 s = make_double2(0.0, 0.0);
#pragma unroll 4
  for (int j = 2 * warp + (lane >> 4); j < n; j += 8)
    if (a < n && j != a) {
      const double2 v = M[(size_t)max(a, j) * N + min(a, j)];
      s.x += v.x;
      s.y += v.y;
    }
  s.x += __shfl_xor_sync(FULL, s.x, 16);
  s.y += __shfl_xor_sync(FULL, s.y, 16);
  if (lane < CS_ATOMS) s_part[group][warp][lane] = s;
  __syncthreads();
  if (warp == 0 && lane < CS_ATOMS && a < N) {
#pragma unroll
    for (int w = 1; w < 4; ++w) {
      s.x += s_part[group][w][lane].x;
      s.y += s_part[group][w][lane].y;
    }
    const size_t at = (size_t)b * N + a;
    c.w.cn[at] = s.x;
    c.w.cnq[at] = s.y;
    if (c.out.d_cn) c.out.d_cn[at] = s.x;
  }
}

}  // namespace

__global__ void __launch_bounds__(128) cn64_sum_kernel(Ctx c) {
  cn64_sum<1>(c, blockIdx.y, CS_ATOMS * blockIdx.x);
}

void launch_cn64_sum(const Ctx &c, cudaStream_t st) {
  cn64_sum_kernel<<<dim3((c.N + CS_ATOMS - 1) / CS_ATOMS, c.B), 128, 0, st>>>(c);
}

// Off-diagonal Coulomb matrix of the real atoms (packed lower rows); CTAs from
// ``ctas`` on add up the coordination numbers.  A thread
// per pair of the flattened triangle, so that small structures fill their
// warps; pairs with g r < 6.6 (beyond, erf = 1 to the last bit) are queued per
// warp and evaluated 32 at a time, so that erf runs with full warps.
__global__ void __launch_bounds__(128) eeq64_build_kernel(Ctx c, int rounds, int ctas) {
  __shared__ int s_i[4][64], s_j[4][64];
  const int b = blockIdx.y;
  if ((int)blockIdx.x >= ctas) {
    cn64_sum<1>(c, b, CS_ATOMS * ((int)blockIdx.x - ctas));
    return;
  }
  const int N = c.N, n = c.w.n_eff[b];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const long long pairs = (long long)n * (n - 1) / 2;
  long long t = ((long long)blockIdx.x * 4 + warp) * 32 * rounds + lane;
  if (t - lane >= pairs) return;
  const size_t ab = (size_t)b * N;
  const int *C = c.w.cidx + ab, *Z = c.w.z + ab;
  const double *P = c.positions + 3 * ab;
  double *L = eeq64_factor(c, b);
  auto pair = [&](int i, int j, bool near) {
    const double dx = P[3 * i] - P[3 * j], dy = P[3 * i + 1] - P[3 * j + 1],
                 dz = P[3 * i + 2] - P[3 * j + 2];
    const double r2 = dx * dx + dy * dy + dz * dz;
    double v = rsqrt(r2);
    if (near) {
      const double ra = c.tab.eeq_rad[Z[i]], rb = c.tab.eeq_rad[Z[j]];
      v *= erf(r2 * v * rsqrt(ra * ra + rb * rb));
      if (!(r2 > 0.0)) v = nan("");  // coincident atoms: erf(0) / 0
    }
    L[tri_index(C[i], C[j])] = v;
  };
  int queued = 0;
  for (int k = 0; k < rounds; ++k, t += 32) {
    int i = 0, j = 0;
    bool near = false;
    if (t < pairs) {
      tri_entry(t, i, j);
      ++i;  // j < i
      if (Z[i] != 0 && Z[j] != 0) {
        const float4 pi = c.w.pos32[ab + i], pj = c.w.pos32[ab + j];
        const float ra = c.w.aux32[ab + i].z, rb = c.w.aux32[ab + j].z;
        const float ex = pi.x - pj.x, ey = pi.y - pj.y, ez = pi.z - pj.z;
        near = !(ex * ex + ey * ey + ez * ez > 44.0f * (ra * ra + rb * rb));
        if (!near) pair(i, j, false);
      }
    }
    const unsigned m = __ballot_sync(FULL, near);
    if (near) {
      const int at = queued + __popc(m & ((1u << lane) - 1u));
      s_i[warp][at] = i;
      s_j[warp][at] = j;
    }
    queued += __popc(m);
    __syncwarp();
    if (queued >= 32) {
      pair(s_i[warp][lane], s_j[warp][lane], true);
      queued -= 32;
      __syncwarp();
      if (lane < queued) {
        s_i[warp][lane] = s_i[warp][32 + lane];
        s_j[warp][lane] = s_j[warp][32 + lane];
      }
      __syncwarp();
    }
  }
  if (lane < queued) pair(s_i[warp][lane], s_j[warp][lane], true);
}

namespace {

// The smooth cap of atom a's EEQ coordination number (and its derivative), in
// place of the raw count; returns the EEQ right-hand side -chi + kcn sqrt(cn).
//   log(1 + e^m) - log(1 + e^(m - cn)) as log1p(expm1(cn) / (1 + e^(cn - m))):
// the same function without the cancellation of the two logarithms, so that
// nearly isolated atoms (cn << 1) keep a relative accuracy (the right-hand
// side takes sqrt(cn), which magnifies absolute noise there).
__device__ __forceinline__ double eeq64_cap(const Ctx &c, size_t a) {
  const double cn = c.w.cnq[a];
  const double f = 1.0 / (1.0 + exp(cn - c.par.cn_eeq_max));
  const double cq = log1p(expm1(cn) * f);
  c.w.cnq[a] = cq;
  c.w.dcnq[a] = f;
  const int z = c.w.z[a];
  return -c.tab.eeq_chi[z] + c.tab.eeq_kcn[z] * (cq > 0.0 ? sqrt(cq) : 0.0);
}

__device__ __forceinline__ double eeq64_diagonal(const Ctx &c, int z) {
  return c.tab.eeq_eta[z] + SQRT_2_OVER_PI / c.tab.eeq_rad[z];
}

}  // namespace

// Capped EEQ coordination numbers of all atoms; with the EEQ, right-hand
// sides and diagonal of its matrix (structures of the multi-CTA path).
__global__ void __launch_bounds__(128) eeq64_rhs_kernel(Ctx c, bool eeq) {
  const size_t a = (size_t)blockIdx.x * 128 + threadIdx.x;
  if (a >= (size_t)c.B * c.N || c.w.z[a] == 0) return;
  const double v = eeq64_cap(c, a);
  if (!eeq) return;
  const int b = (int)(a / c.N), k = c.w.cidx[a];
  eeq64_rhs(c, b, 0)[k] = v;
  eeq64_rhs(c, b, 1)[k] = 1.0;
  eeq64_factor(c, b)[tri_index(k, k)] = eeq64_diagonal(c, c.w.z[a]);
}

// One structure per CTA in shared memory (N <= EEQ64_SMALL, at most 32 S rows
// beside the diagonal block).
template <int S>
__global__ void __launch_bounds__(256) eeq64_small_kernel(Ctx c) {
  extern __shared__ double s_dyn[];
  __shared__ PanelSmem sm;
  __shared__ SolveSmem ss;
  constexpr int CW = 4;
  const int b = blockIdx.x, N = c.N;
  const int m = eeq64_order(c, b);
  double *v = s_dyn;            // 2 x N
  double *L = s_dyn + 2 * N;    // packed
  const int tri_m = m * (m + 1) / 2;
  double *G = eeq64_factor(c, b);
  for (int t = threadIdx.x; t < tri_m; t += blockDim.x) L[t] = G[t];  // (diagonal: below)
  for (int a = 0; a < N; a += 2 * CS_ATOMS) {
    cn64_sum<2>(c, b, a);
    __syncthreads();
  }
  for (int i = threadIdx.x; i < N; i += blockDim.x) {
    const size_t a = (size_t)b * N + i;
    const int k = c.w.cidx[a];
    if (k < 0) continue;
    v[k] = eeq64_cap(c, a);
    v[N + k] = 1.0;
    L[tri_index(k, k)] = eeq64_diagonal(c, c.w.z[a]);
  }
  __syncthreads();
  const int warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
  for (int k0 = 0; k0 < m; k0 += EB) {
    const int kb = min(EB, m - k0), t0 = k0 + kb;
    eeq64_panel<S>(PanelRows{L, nullptr, v, v + N, k0, kb, m}, 0, sm, c.w.status);
    __syncthreads();
    const int T = (m - t0 + 31) / 32;
    constexpr int PARTS = EB / CW;
    for (int t = warp; t < T * (T + 1) / 2 * PARTS; t += nw) {
      int ti, tj;
      tri_entry(t / PARTS, ti, tj);
      eeq64_update_tile<CW>(L, nullptr, v, v + N, ti, tj, t % PARTS, k0, t0, m);
    }
    __syncthreads();
  }
  eeq64_charges(c, b, L, InvAt{L, nullptr}, v, N, m, ss);
  if (c.flags & D4_FLAG_GRADIENT)  // the adjoint solve takes the factor
    for (int t = threadIdx.x; t < tri_m; t += blockDim.x) G[t] = L[t];
}

// Panel at k0 of every structure; a CTA factorises the diagonal block for its
// own 32 S rows (the block's result leaves as the inverse, into the scratch).
template <int S>
__global__ void __launch_bounds__(256) eeq64_panel_kernel(Ctx c, int k0) {
  __shared__ PanelSmem sm;
  const int b = blockIdx.y;
  const int m = eeq64_order(c, b);
  if (k0 >= m) return;
  const PanelRows R{eeq64_factor(c, b), eeq64_inv(c, b) + (size_t)k0 * EB, eeq64_rhs(c, b, 0),
                    eeq64_rhs(c, b, 1), k0, min(EB, m - k0), m};
  const int w0 = blockIdx.x * 32 * S;
  if (w0 < R.count()) eeq64_panel<S>(R, w0, sm, c.w.status);
}

// Trailing update after the panel at k0: a warp per 32 x CW tile.
template <int CW>
__global__ void __launch_bounds__(128) eeq64_update_kernel(Ctx c, int k0) {
  __shared__ double s_j[4][EB * CW];
  constexpr int PARTS = EB / CW;
  const int b = blockIdx.y;
  const int m = eeq64_order(c, b);
  const int t0 = k0 + EB;
  if (t0 >= m) return;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int T = (m - t0 + 31) / 32;
  const int t = blockIdx.x * 4 + warp;
  if (t >= T * (T + 1) / 2 * PARTS) return;
  int ti, tj;
  tri_entry(t / PARTS, ti, tj);
  double *L = eeq64_factor(c, b);
  double *sj = s_j[warp];
#pragma unroll
  for (int q = 0; q < CW; ++q) {
    const int j = t0 + 32 * tj + CW * (t % PARTS) + q;
    sj[lane * CW + q] = j < m ? L[tri_index(j, k0 + lane)] : 0.0;
  }
  __syncwarp();
  eeq64_update_tile<CW>(L, sj, eeq64_rhs(c, b, 0), eeq64_rhs(c, b, 1), ti, tj, t % PARTS, k0,
                        t0, m);
}

// Backward solve, charges, and the block inverses into the factor.  SMEM: the
// vectors in shared memory, else where they are (eeq64_vec_fits).
template <bool SMEM>
__global__ void __launch_bounds__(256) eeq64_finish_kernel(Ctx c) {
  extern __shared__ double s_dyn[];
  __shared__ SolveSmem ss;
  const int b = blockIdx.x, N = c.N;
  const int m = eeq64_order(c, b);
  double *L = eeq64_factor(c, b), *X = eeq64_inv(c, b);
  double *v0 = eeq64_rhs(c, b, 0), *v1 = eeq64_rhs(c, b, 1);
  if (SMEM) {
    for (int t = threadIdx.x; t < m; t += blockDim.x) {
      s_dyn[t] = v0[t];
      s_dyn[N + t] = v1[t];
    }
    v0 = s_dyn;
    v1 = s_dyn + N;
  }
  __syncthreads();
  eeq64_charges(c, b, L, InvAt{L, X}, v0, v1 - v0, m, ss);
  if (c.flags & D4_FLAG_GRADIENT)
    for (int t = threadIdx.x; t < m * EB; t += blockDim.x) {
      const int i = t / EB, cc = t % EB, k0 = i & ~(EB - 1);
      if (k0 + cc <= i) L[tri_index(i, k0 + cc)] = X[(size_t)k0 * EB + (i - k0) * EB + cc];
    }
}

// Adjoint of the constrained EEQ solve: w = A^-1 (g - nu 1) with sum(w) = 0,
// g = dE/dq; as for the charges, nu = z_1 . z_g / z_1 . z_1 and w = L^-T (z_g -
// nu z_1).  Then dE/d(raw EEQ CN) = w kcn / (2 sqrt(cn)) dcap.  SMEM: the vector
// in shared memory, else in the room of the pair records, whose readers are done.
template <bool SMEM>
__global__ void __launch_bounds__(ES_THREADS) eeq64_adjoint_kernel(Ctx c) {
  extern __shared__ double s_dyn[];
  __shared__ SolveSmem ss;
  const int b = blockIdx.x, N = c.N;
  const int m = eeq64_order(c, b);
  const double *L = eeq64_factor(c, b), *z1 = c.w.eeq_y + (size_t)b * N;
  double *v = SMEM ? s_dyn : c.w.pr_r + (size_t)b * N;
  for (int i = threadIdx.x; i < N; i += ES_THREADS) {
    const int k = c.w.cidx[(size_t)b * N + i];
    if (k >= 0) v[k] = c.w.dEdq[(size_t)b * N + i];
  }
  __syncthreads();
  const InvAt inv{L, nullptr};
  eeq64_solve<true>(L, inv, v, m, ss);
  const double su = eeq64_dot(v, z1, m, ss);
  const double nu = m > 0 ? su / c.w.eeq_sum[2 * b] : 0.0;
  for (int k = threadIdx.x; k < m; k += ES_THREADS) v[k] = fma(-nu, z1[k], v[k]);
  __syncthreads();
  eeq64_solve<false>(L, inv, v, m, ss);
  for (int i = threadIdx.x; i < N; i += ES_THREADS) {
    const size_t a = (size_t)b * N + i;
    const int k = c.w.cidx[a];
    double w = 0.0, d = 0.0;
    if (k >= 0) {
      w = v[k];
      const double cq = c.w.cnq[a];
      d = cq > 0.0 ? w * c.tab.eeq_kcn[c.w.z[a]] * 0.5 / sqrt(cq) * c.w.dcnq[a] : 0.0;
    }
    c.w.eeq_w[a] = w;
    c.w.dEdcnq[a] = d;
  }
}

// Whether the final solves' vectors fit a CTA's shared memory (N <= 14080).
static bool eeq64_vec_fits(const Ctx &c) {
  return !(c.flags & D4_FLAG_TEST_FALLBACK) && 16 * (size_t)c.N <= 220 * 1024;
}

template <int S>
static void launch_small(const Ctx &c, cudaStream_t st) {
  const size_t bytes = 8 * (2 * (size_t)c.N + (size_t)c.N * (c.N + 1) / 2);
  ensure_smem(eeq64_small_kernel<S>, bytes);
  eeq64_small_kernel<S><<<c.B, ES_THREADS, bytes, st>>>(c);
}

void launch_eeq64_cap(const Ctx &c, cudaStream_t st, bool eeq) {
  const size_t total = (size_t)c.B * c.N;
  eeq64_rhs_kernel<<<(unsigned)((total + 127) / 128), 128, 0, st>>>(c, eeq);
}

void launch_eeq64(const Ctx &c, cudaStream_t st) {
  const int B = c.B, N = c.N;
  const long long pairs = (long long)N * (N - 1) / 2;
  // eight pairs per thread fill the queues of a batch, one spreads few pairs
  const int rounds = B * pairs <= 4LL * sm_count() * 128 ? 1 : 8;
  const int ctas = (int)((pairs + 128 * rounds - 1) / (128 * rounds));
  // (the one-CTA solver adds up its structure's coordination numbers itself: beside
  // the pairs of many small structures their CTAs cost 12 us of 360 x 30 atoms)
  const int sums = N <= EEQ64_SMALL ? 0 : (N + CS_ATOMS - 1) / CS_ATOMS;
  if (ctas + sums > 0)
    eeq64_build_kernel<<<dim3(ctas + sums, B), 128, 0, st>>>(c, rounds, ctas);
  if (N <= EEQ64_SMALL) {
    const int rows = EB + 2 + (N > EB ? N - EB : 0);  // beside the first diagonal block
    if (rows <= 64)
      launch_small<2>(c, st);
    else if (rows <= 96)
      launch_small<3>(c, st);
    else
      launch_small<4>(c, st);
    return;
  }
  launch_eeq64_cap(c, st, true);
  for (int k0 = 0; k0 < N; k0 += EB) {
    const int left = N > k0 + EB ? N - k0 - EB : 0, rows = EB + 2 + left;
    const int T = (left + 31) / 32;
    // 32 rows per CTA while that leaves SMs idle, 128 once the CTAs' own
    // diagonal factors would crowd the pipe
    if ((long long)B * ((rows + 31) / 32) <= 4 * sm_count())
      eeq64_panel_kernel<1><<<dim3((rows + 31) / 32, B), 256, 0, st>>>(c, k0);
    else
      eeq64_panel_kernel<4><<<dim3((rows + 127) / 128, B), 256, 0, st>>>(c, k0);
    if (T == 0) break;
    const long long tiles = (long long)T * (T + 1) / 2;
    // four columns per warp while that leaves sub-partitions idle
    if (B * tiles * 8 <= 4 * sm_count() * 4)
      eeq64_update_kernel<4><<<dim3((unsigned)(tiles * 8 + 3) / 4, B), 128, 0, st>>>(c, k0);
    else
      eeq64_update_kernel<8><<<dim3((unsigned)(tiles * 4 + 3) / 4, B), 128, 0, st>>>(c, k0);
  }
  if (eeq64_vec_fits(c)) {
    ensure_smem(eeq64_finish_kernel<true>, 16 * (size_t)N);
    eeq64_finish_kernel<true><<<B, ES_THREADS, 16 * (size_t)N, st>>>(c);
  } else {
    eeq64_finish_kernel<false><<<B, ES_THREADS, 0, st>>>(c);
  }
}

void launch_eeq64_adjoint(const Ctx &c, cudaStream_t st) {
  if (eeq64_vec_fits(c)) {
    ensure_smem(eeq64_adjoint_kernel<true>, 8 * (size_t)c.N);
    eeq64_adjoint_kernel<true><<<c.B, ES_THREADS, 8 * (size_t)c.N, st>>>(c);
  } else {
    eeq64_adjoint_kernel<false><<<c.B, ES_THREADS, 0, st>>>(c);
  }
}

}  // namespace d4
