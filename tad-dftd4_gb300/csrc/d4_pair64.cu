// FP64 pair stages of the plain method for the common case (rational damping,
// unit energy weights, approximate C9): everything a pair needs is evaluated
// once per unordered pair, a thread each, and leaves as numbers per pair;
// kernels with a warp per atom then only sum rows.  A warp instruction takes
// 64 cycles of its sub-partition's FP64 pipe, so what counts is the number of
// FP64 instructions per pair and full warps; loads hide behind it.
//
// Where the pair numbers live (i < j): pr4[i][j] the ATM record, pr_S[i][j]
// dE/d(r^2), pr_S[j][i] dE/dC6, pr_P[i][j] the ATM energy sum (cleared here),
// pr_P[j][i] 1 / (2 C6(q=0)).  e3 and pgrad are the output arrays themselves.
//
// Measured, 64 structures of 8..200 atoms / 360 of 30 atoms / 57 atoms (us;
// before: a warp per atom over ordered pairs, d4_fp64.cu):
//   C6, two-body term, records   566 / 337 / 58 -> 197 / 71 / 17
//   C6 adjoints, chain rule      189 / 188 / 30 -> 133 / 71 / 14
//   CN / EEQ adjoints, forces    455 / 153 / 35 -> 186 / 92 / 20
#include "d4_common.cuh"
#include "d4_fpmath.cuh"
#include "d4_kernels.cuh"

namespace d4 {

namespace {

constexpr int TB = 64;   // atoms per block of the pair kernel's tiles
constexpr int PT = 128;  // threads of its CTAs

}  // namespace

// C6 at the charges and at q = 0, the BJ two-body energy, its derivatives with
// respect to r^2, C6 and the parameters, and the ATM record of every pair i <
// j.  A CTA takes `per` pairs of a tile of two 64-atom blocks (a triangle on
// the diagonal), numbered so that no lane idles; the weighted polarisabilities
// of the tile's atoms are staged in shared memory (D4; D4S picks the partner's
// slot and reads them directly).
template <bool D4S>
__global__ void __launch_bounds__(PT) pair64_kernel(Ctx c, int per, int parts) {
  extern __shared__ double s_a[];  // [2 blocks][TB][2 NFREQ], with (3 / pi) w on the first
  __shared__ double s_sr[2][TB];   // sqrt(3 r4r2)
  const int b = blockIdx.y, N = c.N, n = c.w.n_eff[b];
  const int tile = blockIdx.x / parts, part = blockIdx.x % parts;
  int J, I;
  tri_entry(tile, J, I);
  const int i0 = TB * I, j0 = TB * J;
  if (j0 >= n) return;
  const int ni = min(TB, n - i0), nj = min(TB, n - j0);
  const int count = I == J ? ni * (ni - 1) / 2 : ni * nj;
  const int first = part * per;
  if (first >= count) return;
  const d4_params_t &p = c.par;
  const size_t ab = (size_t)b * N;
  if (!D4S) {
    for (int t = threadIdx.x; t < (ni + nj) * NFREQ; t += PT) {
      const int a = t / NFREQ, w = t % NFREQ;
      const int side = a >= ni, k = side ? a - ni : a;
      const size_t o = (ab + (side ? j0 : i0) + k) * NFREQ + w;
      const double f = side ? 1.0 : THOPI * c.tab.freq_weights[w];
      double *d = s_a + ((size_t)(side * TB + k) * 2) * NFREQ + w;
      d[0] = f * c.w.A[o];
      d[NFREQ] = f * c.w.A0[o];
    }
  }
  for (int t = threadIdx.x; t < ni + nj; t += PT) {
    const int side = t >= ni, k = side ? t - ni : t;
    const size_t a = ab + (side ? j0 : i0) + k;
    const int z = c.w.z[a];
    s_sr[side][k] = z != 0 ? sqrt(3.0 * atom_r4r2(c, a, z)) : 0.0;
  }
  __syncthreads();
  const bool grad = (c.flags & D4_FLAG_GRADIENT) != 0;
  const bool pgrad = (c.flags & D4_FLAG_PARAM_GRAD) != 0;
  const double *P = c.positions + 3 * ab;
  const size_t base = ab * N;
  const double alp3 = p.alp / 3.0;
  double pg[5] = {0.0, 0.0, 0.0, 0.0, 0.0};
  for (int t = first + threadIdx.x; t < min(count, first + per); t += PT) {
    int li, lj;
    if (I == J) {
      tri_entry(t, lj, li);
      ++lj;  // li < lj
    } else {
      li = t / nj;
      lj = t % nj;
    }
    const int i = i0 + li, j = j0 + lj;
    const size_t up = base + (size_t)i * N + j, lo = base + (size_t)j * N + i;
    if (c.w.z[ab + i] == 0 || c.w.z[ab + j] == 0) {  // padding: a pair of nothing
      c.w.pr4[up] = PairRec{0.0, 0.0, 0.0, 0.0};
      if (grad) c.w.pr_S[up] = c.w.pr_S[lo] = c.w.pr_P[up] = c.w.pr_P[lo] = 0.0;
      if (pgrad) c.w.pr_da1[up] = c.w.pr_da1[lo] = c.w.pr_da2[up] = 0.0;
      continue;
    }
    const double dx = P[3 * i] - P[3 * j], dy = P[3 * i + 1] - P[3 * j + 1],
                 dz = P[3 * i + 2] - P[3 * j + 2];
    const double r2 = dx * dx + dy * dy + dz * dz;
    double c6 = 0.0, c60 = 0.0;
    if (D4S) {
      const size_t oi = ((ab + i) * c.S + c.w.slot[ab + j]) * NFREQ;
      const size_t oj = ((ab + j) * c.S + c.w.slot[ab + i]) * NFREQ;
#pragma unroll
      for (int w = 0; w < NFREQ; ++w) {
        const double f = THOPI * c.tab.freq_weights[w];
        c6 = fma(f * c.w.A[oi + w], c.w.A[oj + w], c6);
        c60 = fma(f * c.w.A0[oi + w], c.w.A0[oj + w], c60);
      }
    } else {
      const double *ai = s_a + (size_t)li * 2 * NFREQ;
      const double *aj = s_a + (size_t)(TB + lj) * 2 * NFREQ;
#pragma unroll
      for (int w = 0; w < NFREQ; ++w) {
        c6 = fma(ai[w], aj[w], c6);
        c60 = fma(ai[NFREQ + w], aj[NFREQ + w], c60);
      }
    }
    const double sqq = s_sr[0][li] * s_sr[1][lj] * (1.0 / 1.7320508075688772935);
    const double R0 = fma(p.a1, sqq, p.a2);
    const double ir = rsqrt(r2), u = ir * ir;
    const double y60 = c60 > 0.0 ? rsqrt_pos(c60) : 0.0;
    const double L = log(R0 * ir);
    c.w.pr4[up] = PairRec{r2, u, pair_t(alp3 * L), c60 * y60 * (u * ir)};
    double e = 0.0, S = 0.0, K = 0.0;
    if (r2 <= c.cut2_sq) {
      const double qq = sqq * sqq;
      const double r4 = r2 * r2, r6 = r4 * r2, R02 = R0 * R0, R06 = R02 * R02 * R02;
      const double t6 = rcp_pos(r6 + R06);
      double h = p.s6 * t6;             // e = c6 h
      double g = 3.0 * h * t6 * r4;     // -dh/d(r^2)
      double gR = 6.0 * h * t6 * R06;   // -R0 dh/dR0
      pg[0] = fma(c6, t6, pg[0]);
      if (p.has_s8) {
        const double t8 = rcp_pos(fma(r6, r2, R06 * R02));
        const double q8 = qq * t8, h8 = p.s8 * q8;
        h += h8;
        g = fma(4.0 * h8 * t8, r6, g);
        gR = fma(8.0 * h8 * t8, R06 * R02, gR);
        pg[1] = fma(c6, q8, pg[1]);
      }
      if (p.has_s10) {
        const double R010 = R06 * R02 * R02;
        const double t10 = rcp_pos(fma(r6, r4, R010));
        const double q10 = qq * qq * (49.0 / 40.0) * t10, h10 = p.s10 * q10;
        h += h10;
        g = fma(5.0 * h10 * t10, r6 * r2, g);
        gR = fma(10.0 * h10 * t10, R010, gR);
        pg[2] = fma(c6, q10, pg[2]);
      }
      e = -0.5 * c6 * h;  // half of the pair energy each
      S = c6 * g;
      K = -h;
      if (pgrad) {
        const double dR = c6 * gR / R0;
        pg[3] = fma(dR, sqq, pg[3]);
        pg[4] += dR;
      }
      atomicAdd(&c.w.e3[ab + i], e);
      atomicAdd(&c.w.e3[ab + j], e);
    }
    if (grad) {
      c.w.pr_S[up] = S;
      c.w.pr_S[lo] = K;
      c.w.pr_P[up] = 0.0;
      c.w.pr_P[lo] = 0.5 * y60 * y60;
    }
    if (pgrad) {
      const double iR = 1.0 / R0;
      c.w.pr_da1[up] = sqq * iR;
      c.w.pr_da2[up] = iR;
      c.w.pr_da1[lo] = L;
    }
    // the largest r^2 of both atoms: non-negative doubles order as their bits
    if (r2 > c.cut3_sq) {
      atomicMax((unsigned long long *)&c.w.rowmax[ab + i], __double_as_longlong(r2));
      atomicMax((unsigned long long *)&c.w.rowmax[ab + j], __double_as_longlong(r2));
    }
  }
  if (pgrad) {
    const double sign[5] = {-1.0, -1.0, -1.0, 1.0, 1.0};
#pragma unroll
    for (int k = 0; k < 5; ++k) {
      pg[k] = warp_sum(pg[k]);
      if ((threadIdx.x & 31) == 0)
        atomicAdd(&c.w.pgrad[b * D4_PARAM_GRAD_STRIDE + k], sign[k] * pg[k]);
    }
  }
}

namespace {

// Sums over the warp of 24 values per lane, scattered: lane 16 b4 + 8 b3 + 4
// b2 + 2 b1 + b0 ends with the sum of value 12 b4 + 6 b3 + 3 b2 + 2 b1 + b0
// (nothing for b1 = b0 = 1).  24 additions instead of 120.
__device__ __forceinline__ double reduce_scatter24(double (&v)[24]) {
  const int lane = threadIdx.x & 31;
  auto halve = [&](int h, int m) {
    const bool up = (lane & h) != 0;
#pragma unroll
    for (int q = 0; q < 12; ++q)
      if (q < m) {
        const double keep = up ? v[q + m] : v[q], send = up ? v[q] : v[q + m];
        v[q] = keep + __shfl_xor_sync(0xffffffffu, send, h);
      }
  };
  halve(16, 12);
  halve(8, 6);
  halve(4, 3);
  v[3] = 0.0;
  halve(2, 2);
  halve(1, 1);
  return v[0];
}
__device__ __forceinline__ int reduce_scatter24_index() {
  const int l = threadIdx.x & 31;
  const int k = (l & 16 ? 12 : 0) + (l & 8 ? 6 : 0) + (l & 4 ? 3 : 0) + (l & 3);
  return (l & 3) == 3 ? -1 : k;
}

constexpr int BX = 4;  // atoms (warps) per CTA of pair64_bwd_kernel

}  // namespace

// dE/dA and dE/dA0 of atom x from dE/dC6 and the ATM energy sums, the chain
// rule to CN and q, and the ATM part of its energy (a sixth of its pair
// sums, d4_atm64.cu).  A warp per atom; D4 stages 32 partners' weighted
// polarisabilities at a time in shared memory.
template <bool D4S>
__global__ void __launch_bounds__(32 * BX) pair64_bwd_kernel(Ctx c) {
  __shared__ double s_a[D4S ? 1 : 32 * 2 * NFREQ];
  __shared__ double2 s_kd[D4S ? 1 : BX][32];  // dE/dC6 and its like at q = 0 of the partners
  const int b = blockIdx.y, N = c.N, n = c.w.n_eff[b];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int x = blockIdx.x * BX + warp;
  const size_t ab = (size_t)b * N;
  if ((int)blockIdx.x * BX >= n) {
    if (x < N && lane == 0) c.w.dEdcn[ab + x] = c.w.dEdq[ab + x] = 0.0;
    return;
  }
  const bool live = x < n && c.w.z[ab + x] != 0;
  const size_t ax = ab + min(x, N - 1);
  const size_t base = ab * N;
  const int nslot = D4S ? c.w.n_slots[b] : 1;
  const int slot_x = D4S ? c.w.slot[ax] : 0;
  double psum = 0.0, dcn = 0.0, dq = 0.0;
  // Few partners: a lane per frequency, the partners in turn (two FMAs each);
  // else a lane per partner (46 FMAs per 32 of them and 48 additions to sum up).
  if (!D4S && 2 * n <= 46 * ((n + 31) / 32) + 48) {
    double g = 0.0, g0 = 0.0;
    for (int y0 = 0; y0 < n; y0 += 32) {
      __syncthreads();
      const int ny = min(32, n - y0), y = y0 + lane;
      for (int t = threadIdx.x; t < ny * NFREQ; t += 32 * BX) {
        const int k = t / NFREQ, w = t % NFREQ;
        s_a[2 * k * NFREQ + w] = c.w.A[(ab + y0 + k) * NFREQ + w];
        s_a[(2 * k + 1) * NFREQ + w] = c.w.A0[(ab + y0 + k) * NFREQ + w];
      }
      double2 kd = make_double2(0.0, 0.0);
      if (live && y < n && y != x && c.w.z[ab + y] != 0) {
        const size_t lo = (size_t)min(x, y), hi = (size_t)max(x, y);
        const double Pv = c.w.pr_P[base + lo * N + hi];
        kd.x = c.w.pr_S[base + hi * N + lo];
        kd.y = Pv != 0.0 ? Pv * c.w.pr_P[base + hi * N + lo] : 0.0;
        psum += Pv;
      }
      s_kd[warp][lane] = kd;
      __syncthreads();
      const double *A = s_a + min(lane, NFREQ - 1);
#pragma unroll 8
      for (int k = 0; k < ny; ++k) {
        const double2 v = s_kd[warp][k];
        g = fma(v.x, A[2 * k * NFREQ], g);
        g0 = fma(v.y, A[(2 * k + 1) * NFREQ], g0);
      }
    }
    if (live && lane < NFREQ) {
      const size_t o = ax * NFREQ + lane;
      const double f = THOPI * c.tab.freq_weights[lane];
      dcn = f * (g * c.w.dA_dcn[o] + g0 * c.w.dA0_dcn[o]);
      dq = f * g * c.w.dA_dq[o];
    }
  } else {
    for (int s = 0; s < nslot; ++s) {
      double g[24], g0[24];
#pragma unroll
      for (int w = 0; w < 24; ++w) g[w] = g0[w] = 0.0;
      for (int y0 = 0; y0 < n; y0 += 32) {
        if (!D4S) {
          __syncthreads();
          const int ny = min(32, n - y0);
          for (int t = threadIdx.x; t < ny * NFREQ; t += 32 * BX) {
            const int k = t / NFREQ, w = t % NFREQ;
            s_a[2 * k * NFREQ + w] = c.w.A[(ab + y0 + k) * NFREQ + w];
            s_a[(2 * k + 1) * NFREQ + w] = c.w.A0[(ab + y0 + k) * NFREQ + w];
          }
          __syncthreads();
        }
        const int y = y0 + lane;
        if (!live || y >= n || y == x || c.w.z[ab + y] == 0) continue;
        if (D4S && c.w.slot[ab + y] != s) continue;
        const size_t lo = (size_t)min(x, y), hi = (size_t)max(x, y);
        const double K = c.w.pr_S[base + hi * N + lo];
        const double Pv = c.w.pr_P[base + lo * N + hi];
        const double D = Pv != 0.0 ? Pv * c.w.pr_P[base + hi * N + lo] : 0.0;
        psum += Pv;
        const double *A, *A0;
        if (D4S) {
          const size_t o = ((ab + y) * c.S + slot_x) * NFREQ;
          A = c.w.A + o;
          A0 = c.w.A0 + o;
        } else {
          A = s_a + 2 * lane * NFREQ;
          A0 = A + NFREQ;
        }
#pragma unroll
        for (int w = 0; w < NFREQ; ++w) {
          g[w] = fma(K, A[w], g[w]);
          g0[w] = fma(D, A0[w], g0[w]);
        }
      }
      const double gw = reduce_scatter24(g), gw0 = reduce_scatter24(g0);
      const int w = reduce_scatter24_index();
      if (live && w >= 0 && w < NFREQ) {
        const size_t o = (ax * c.S + s) * NFREQ + w;
        const double f = THOPI * c.tab.freq_weights[w];
        dcn += f * (gw * c.w.dA_dcn[o] + gw0 * c.w.dA0_dcn[o]);
        dq += f * gw * c.w.dA_dq[o];
      }
    }
  }
  dcn = warp_sum(dcn);
  dq = warp_sum(dq);
  psum = warp_sum(psum);
  if (lane == 0 && x < N) {
    c.w.dEdcn[ax] = dcn;
    c.w.dEdq[ax] = dq;
    if (live) c.w.e3[ax] += psum * (1.0 / 6.0);
  }
}

// dE/d(r^2) through the D4 CN, the EEQ CN and the EEQ Coulomb matrix, added to
// pr_S, a thread per pair i < j.  A pair needs exp and erf only where a
// counting function or 1 - erf is left (x <= 9: 1/2 erfc(9) < 1e-36; g r <=
// 6.6: the terms beyond are below 2^-55 of the pair's Coulomb term): those are
// queued per warp and evaluated 32 at a time, so that the FP64 instructions
// run with full warps.
__global__ void __launch_bounds__(PT) pair64_cn_bwd_kernel(Ctx c, int rounds) {
  __shared__ int s_i[PT / 32][64], s_j[PT / 32][64];
  const int b = blockIdx.y, N = c.N, n = c.w.n_eff[b];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const long long pairs = (long long)n * (n - 1) / 2;
  long long t = ((long long)blockIdx.x * (PT / 32) + warp) * 32 * rounds + lane;
  if (t - lane >= pairs) return;
  const d4_params_t &p = c.par;
  const bool eeq = (c.flags & D4_FLAG_CHARGES_IN) == 0;
  const size_t ab = (size_t)b * N;
  const double *P = c.positions + 3 * ab;
  const int *Z = c.w.z + ab;
  const float kcn32 = (float)p.kcn;
  double *S = c.w.pr_S + ab * N;
  auto geometry = [&](int i, int j, double &r2, double &ir) {
    const double dx = P[3 * i] - P[3 * j], dy = P[3 * i + 1] - P[3 * j + 1],
                 dz = P[3 * i + 2] - P[3 * j + 2];
    r2 = dx * dx + dy * dy + dz * dz;
    ir = r2 > 0.0 ? rsqrt_pos(r2) : INFINITY;
  };
  const double ik6 = 1.0 / p.k6;
  auto charges = [&](int i, int j) {
    return c.w.eeq_w[ab + i] * c.w.q[ab + j] + c.w.eeq_w[ab + j] * c.w.q[ab + i];
  };
  auto near_pair = [&](int i, int j) {
    double r2, ir;
    geometry(i, j, r2, ir);
    const double r = r2 * ir;
    const int zi = Z[i], zj = Z[j];
    const double ir0 = rcp_pos(c.tab.cov_d3[zi] + c.tab.cov_d3[zj]);
    double dEdr = 0.0;
    double gcn = 0.0;
    if (r2 <= c.cutcn_sq) {  // (en_factor with 1 / k6)
      const double t = fabs(c.tab.en[zi] - c.tab.en[zj]) + p.k5;
      gcn = (c.w.dEdcn[ab + i] + c.w.dEdcn[ab + j]) * (p.k4 * exp(-(t * t) * ik6));
    }
    if (eeq) {
      if (r2 <= c.cutq_sq) gcn += c.w.dEdcnq[ab + i] + c.w.dEdcnq[ab + j];
      const double ra = c.tab.eeq_rad[zi], rb = c.tab.eeq_rad[zj];
      const double g = rsqrt_pos(ra * ra + rb * rb), gr = g * r;
      const double dA = (2.0 * INV_SQRT_PI * exp(-gr * gr) * gr - erf(gr)) * (ir * ir);
      dEdr = -charges(i, j) * dA;
    }
    const double x = p.kcn * (r * ir0 - 1.0);  // erf_count_dr with 1 / r0
    dEdr = fma(gcn, -p.kcn * ir0 * INV_SQRT_PI * exp(-x * x), dEdr);
    S[(size_t)i * N + j] += 0.5 * dEdr * ir;
  };
  int queued = 0;
  for (int k = 0; k < rounds; ++k, t += 32) {
    int i = 0, j = 0;
    bool near = false;
    if (t < pairs) {
      tri_entry(t, j, i);
      ++j;  // i < j
      if (Z[i] != 0 && Z[j] != 0) {
        const float4 pi = c.w.pos32[ab + i], pj = c.w.pos32[ab + j];
        const float4 xi = c.w.aux32[ab + i], xj = c.w.aux32[ab + j];
        const float ex = pi.x - pj.x, ey = pi.y - pj.y, ez = pi.z - pj.z;
        const float r2f = ex * ex + ey * ey + ez * ez;
        near = kcn32 * (sqrtf(r2f) / (xi.x + xj.x) - 1.0f) <= 9.0f ||
               (eeq && r2f <= 44.0f * (xi.z * xi.z + xj.z * xj.z));
        if (!near && eeq) {  // erf = 1: dA/dr = -1 / r^2
          double r2, ir;
          geometry(i, j, r2, ir);
          S[(size_t)i * N + j] += 0.5 * charges(i, j) * (ir * ir * ir);
        }
      }
    }
    const unsigned m = __ballot_sync(0xffffffffu, near);
    if (near) {
      const int at = queued + __popc(m & ((1u << lane) - 1u));
      s_i[warp][at] = i;
      s_j[warp][at] = j;
    }
    queued += __popc(m);
    __syncwarp();
    if (queued >= 32) {
      near_pair(s_i[warp][lane], s_j[warp][lane]);
      queued -= 32;
      __syncwarp();
      if (lane < queued) {
        s_i[warp][lane] = s_i[warp][32 + lane];
        s_j[warp][lane] = s_j[warp][32 + lane];
      }
      __syncwarp();
    }
  }
  if (lane < queued) near_pair(s_i[warp][lane], s_j[warp][lane]);
}

// Gradient of atom i: sum_j 2 dE/d(r_ij^2) (r_i - r_j).  A warp per atom.
__global__ void __launch_bounds__(128) pair64_force_kernel(Ctx c) {
  const int b = blockIdx.y, N = c.N, n = c.w.n_eff[b];
  const int lane = threadIdx.x & 31;
  const int i = blockIdx.x * 4 + (threadIdx.x >> 5);
  if (i >= N) return;
  const size_t ab = (size_t)b * N;
  double gx = 0.0, gy = 0.0, gz = 0.0;
  if (i < n && c.w.z[ab + i] != 0) {
    const double *P = c.positions + 3 * ab, *S = c.w.pr_S + ab * N;
    const double xi = P[3 * i], yi = P[3 * i + 1], zi = P[3 * i + 2];
    for (int j = lane; j < n; j += 32) {
      if (j == i || c.w.z[ab + j] == 0) continue;
      const double s = S[(size_t)min(i, j) * N + max(i, j)];
      gx = fma(s, xi - P[3 * j], gx);
      gy = fma(s, yi - P[3 * j + 1], gy);
      gz = fma(s, zi - P[3 * j + 2], gz);
    }
  }
  gx = warp_sum(gx);
  gy = warp_sum(gy);
  gz = warp_sum(gz);
  if (lane == 0) {
    double *g = c.out.d_gradient + 3 * (ab + i);
    g[0] = 2.0 * gx;
    g[1] = 2.0 * gy;
    g[2] = 2.0 * gz;
  }
}

void launch_pair64(const Ctx &c, cudaStream_t st) {
  const int B = c.B, N = c.N;
  const long long nb = (N + TB - 1) / TB, tiles = nb * (nb + 1) / 2;
  // a pair per thread while that leaves sub-partitions idle, else four
  const long long pairs = (long long)B * N * (N - 1) / 2;
  const int per = pairs <= 4LL * sm_count() * PT ? PT : 4 * PT;
  const int most = N <= TB ? N * (N - 1) / 2 : TB * TB;
  const int parts = most > per ? (most + per - 1) / per : 1;
  const dim3 grid((unsigned)(tiles * parts), B);
  if (c.S > 1 || c.cfg.kind == D4_MODEL_D4S) {
    pair64_kernel<true><<<grid, PT, 0, st>>>(c, per, parts);
  } else {
    const size_t bytes = 8 * (size_t)2 * TB * 2 * NFREQ;
    ensure_smem(pair64_kernel<false>, bytes);
    pair64_kernel<false><<<grid, PT, bytes, st>>>(c, per, parts);
  }
}

void launch_pair64_bwd(const Ctx &c, cudaStream_t st) {
  const dim3 grid((c.N + BX - 1) / BX, c.B);
  if (c.S > 1 || c.cfg.kind == D4_MODEL_D4S)
    pair64_bwd_kernel<true><<<grid, 32 * BX, 0, st>>>(c);
  else
    pair64_bwd_kernel<false><<<grid, 32 * BX, 0, st>>>(c);
}

void launch_pair64_forces(const Ctx &c, cudaStream_t st) {
  const int B = c.B, N = c.N;
  const long long pairs = (long long)N * (N - 1) / 2;
  const int rounds = B * pairs <= 4LL * sm_count() * PT ? 1 : 8;
  const long long per = (long long)PT * rounds;
  if (pairs > 0)
    pair64_cn_bwd_kernel<<<dim3((unsigned)((pairs + per - 1) / per), B), PT, 0, st>>>(c, rounds);
  pair64_force_kernel<<<dim3((N + 3) / 4, B), 128, 0, st>>>(c);
}

}  // namespace d4
