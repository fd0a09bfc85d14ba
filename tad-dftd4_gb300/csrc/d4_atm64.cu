// Register-tiled FP64 ATM of the plain method: all triples i < j < k of
// structures with unit energy weights (any size, padding atoms anywhere).
//
// A warp instruction occupies its sub-partition's FP64 pipe for 64 cycles, so
// everything else (loads, shuffles, integer work, reductions at L2) hides
// behind the FP64 instructions: the kernel is built for the
// fewest FP64 instructions per triple.  The pair records carry r^2, 1/r^2,
// (R0/r)^(alp/3) and sqrt(C6(q=0)) / r^3, so that damping and C9 / R^3 are
// products (no exp per triple), the atom energies follow from the pair
// energy sums, and the (i, k) and (j, k) sums live in registers: ~40 FP64
// instructions per triple with its gradient against ~186 of the per-triple
// kernel (d4_fp64.cu, atm_kernel: one pair (j, k) per lane, an exp, a
// division and full warp sums per triple).  Measured, ATM stage: 64
// structures of 8..200 atoms 11.06 -> 1.76 ms, 360 of 30 atoms 1.36 -> 0.22
// ms, 301 atoms 4.82 -> 0.43 ms, 57 atoms 0.48 -> 0.018 ms (energy +
// gradient); 32 atoms, energy only, 0.125 -> 0.016 ms.  Of the middle atoms'
// order: tiles counted from the last atom instead of the first, and steps
// without the middle atoms below all inner ones, took 1.96 -> 1.76 ms and 0.31
// -> 0.22 ms.
#include "d4_common.cuh"
#include "d4_fpmath.cuh"
#include "d4_kernels.cuh"

namespace d4 {

namespace {

constexpr int A6_K = 8;  // outer atoms per task (lanes of a group)

// Sum of two lanes' values, split: the lane whose bit h is clear keeps the
// sum of the pair's a, the other the sum of the pair's b.
__device__ __forceinline__ double lane_split(double a, double b, int h) {
  const bool up = ((threadIdx.x & 31) & h) != 0;
  const double keep = up ? b : a, send = up ? a : b;
  return keep + __shfl_xor_sync(0xffffffffu, send, h);
}

// (i, j) sums of J middle atoms over the eight lanes of a group, formed as
// the values arrive in bit-reversed order so that few stay live: lane l ends
// with the sum of value l (J = 8), or of value l >> 1 split into halves that
// one more exchange joins (J = 4; both lanes of the pair hold the sum).
template <int J>
struct GroupSum {
  double a, b, c;
  __device__ __forceinline__ void put(int s, double v) {  // s: position in the order of ord()
    if (J == 8) {
      switch (s) {
        case 0: a = v; break;
        case 1: a = lane_split(a, v, 4); break;
        case 2: b = v; break;
        case 3: b = lane_split(b, v, 4); a = lane_split(a, b, 2); break;
        case 4: b = v; break;
        case 5: b = lane_split(b, v, 4); break;
        case 6: c = v; break;
        default: c = lane_split(c, v, 4); b = lane_split(b, c, 2); a = lane_split(a, b, 1);
      }
    } else {
      switch (s) {
        case 0: a = v; break;
        case 1: a = lane_split(a, v, 4); break;
        case 2: b = v; break;
        default:
          b = lane_split(b, v, 4);
          a = lane_split(a, b, 2);
          a += __shfl_xor_sync(0xffffffffu, a, 1);
      }
    }
  }
  __device__ __forceinline__ static constexpr int ord(int s) {  // value put at position s
    constexpr int o8[8] = {0, 4, 2, 6, 1, 5, 3, 7};
    constexpr int o4[4] = {0, 2, 1, 3};
    return J == 8 ? o8[s] : o4[s & 3];
  }
  __device__ __forceinline__ static int mine() {  // index of the value this lane ends with
    const int l = threadIdx.x & 7;
    return J == 8 ? l : l >> 1;
  }
  __device__ __forceinline__ static bool owner() { return J == 8 || (threadIdx.x & 1) == 0; }
};

struct A6 {
  const PairRec *__restrict__ T;
  const double *__restrict__ da1, *__restrict__ da2;  // PGRAD (da1[j][i], j > i: log(R0/r))
  double *S, *P, *e3;
  double cut2, alp6, s9;
  int n, N;
};

struct A6Pg {
  double s9 = 0.0, alp = 0.0, a1 = 0.0, a2 = 0.0;
};

// One step: inner atom i of this lane's group against the J middle atoms
// j0 .. of the task and the lane's outer atom k.  ib: the first group's inner
// atom.  GUARD: some (i, j) are not pairs of the task (i >= j, i beyond the
// range).  MASK: an atom of the
// step has a pair beyond the cutoff, so each triple takes its weight
// (1, 1/3 or 0) and the 1/3 triples their energy attribution.
template <int J, bool GRAD, bool PGRAD, bool GUARD, bool MASK>
__device__ __forceinline__ void a6_step(const A6 &a, int j0, int k, bool kok, int ib, int i,
                                        bool iok, const double (&zjk)[J], const double (&ujk)[J],
                                        const double (&tjk)[J], const double (&qjk)[J],
                                        double (&Sjk)[J], double (&Pjk)[J], double (&Wjk)[J],
                                        double &Ek, A6Pg &pg) {
  const PairRec zero{0.0, 0.0, 0.0, 0.0};
  const PairRec *Ti = a.T + (size_t)(iok ? i : 0) * a.N;
  const bool lk = iok && kok && k > i;
  const PairRec ik = lk ? Ti[k] : zero;
  const double y = ik.x, uy = 0.375 * ik.u;
  const bool fik = !MASK || y <= a.cut2;
  double Sik = 0.0, Pik = 0.0, Wik = 0.0;
  GroupSum<J> gS, gP, gW;
#pragma unroll
  for (int s = 0; s < J; ++s) {
    const int t = GroupSum<J>::ord(s);
    if (GUARD && j0 + t <= ib) {  // no lane of the warp has a triple
      if (GRAD) {
        gS.put(s, 0.0);
        gP.put(s, 0.0);
        if (PGRAD) gW.put(s, 0.0);
      }
      continue;
    }
    PairRec ij;
    if (GUARD) {
      const int jt = j0 + t;
      const bool ok = iok && jt > i;
      ij = ok ? Ti[ok ? jt : 0] : zero;
    } else {
      ij = Ti[j0 + t];
    }
    double x = ij.x, yy = y, z = zjk[t], q = ij.q;
    bool fij = true, fjk = true;
    int m = 3;
    if (MASK) {  // weight 1, 1/3 or 0, folded into C9 / R^3
      fij = x <= a.cut2;
      fjk = z <= a.cut2;
      m = (int)fij + (int)fik + (int)fjk;
      if (GRAD && m == 2) q *= 1.0 / 3.0;
      if (m < 2) q = x = yy = z = 0.0;  // no energy, and no overflow of far pairs
    }
    // R = r_ij r_ik r_jk: w = 3/8 / R^2, ang = w ABC + 1 (times 1/R^3 in D)
    const double w = ij.u * (uy * ujk[t]);
    const double d = x - yy;
    const double A = d + z, B = fma(2.0, x, -A), C = z - d;
    const double AB = A * B;
    const double g = fma(AB * C, w, 1.0);
    // (tjk carries the factor 6: 1 .. 6e300)
    const double fd = rcp_pos<false>(fma(ij.t, ik.t * tjk[t], 1.0));
    const double D = q * (ik.q * qjk[t]) * fd;
    const double e = D * g;
    if (!GRAD) {
      // atom energies in units of e/3: m = 3 gives every atom 1; m = 2 nothing
      // to the atom of both inside pairs and 1/2 to the other two
      if (MASK && m == 2) {
        const double h = 0.5 * e;
        Pik += fjk ? h : 0.0;           // atom i (opposite side jk inside)
        Ek += fij ? h : 0.0;
        Pjk[t] += fik ? h : 0.0;
      } else {
        Pik += e;
        if (MASK) Ek += e;
        Pjk[t] += e;
      }
      continue;
    }
    if (MASK && m == 2 && e != 0.0) {
      // weighted pair sums alone give each atom e_w / 3; wanted are 0 for the
      // atom of both inside pairs and e_w / 2 for the others
      const double es = PGRAD ? e * a.s9 : e;
      const double lo = es * (-1.0 / 3.0), hi = es * (1.0 / 6.0);
      atomicAdd(&a.e3[i], fjk ? hi : lo);
      atomicAdd(&a.e3[j0 + t], fik ? hi : lo);
      atomicAdd(&a.e3[k], fij ? hi : lo);
    }
    // e = Q fd ang with dS/dx = AC + BC - AB and so on; U = Q fd w,
    // V = Q fd (1 + ang (alp/6 (1 - fd) - 5/2))
    const double AC = A * C, BC = B * C;
    const double sm = AB + AC, df = AB - AC;
    const double U = D * w;
    const double V = fma(e, fma(-a.alp6, fd, a.alp6 - 2.5), D);
    Sik = fma(V, ik.u, fma(U, sm - BC, Sik));
    Sjk[t] = fma(V, ujk[t], fma(U, df + BC, Sjk[t]));
    Pik += e;
    Pjk[t] += e;
    gS.put(s, fma(U, BC - df, V * ij.u));
    gP.put(s, e);
    if (PGRAD) {
      const double wv = fma(-e, fd, e);  // e (1 - fd): -dE/d(alp/3 log(R0/r)) of each pair
      Wik += wv;
      Wjk[t] += wv;
      gW.put(s, wv);
    }
  }
  if (!GRAD) {
    if (!MASK) Ek += Pik;
    double ei = Pik;  // over the eight lanes of the group
    ei += __shfl_xor_sync(0xffffffffu, ei, 1);
    ei += __shfl_xor_sync(0xffffffffu, ei, 2);
    ei += __shfl_xor_sync(0xffffffffu, ei, 4);
    if (iok && (threadIdx.x & 7) == 0 && ei != 0.0) atomicAdd(&a.e3[i], ei * (a.s9 / 3.0));
    return;
  }
  const double sc = PGRAD ? a.s9 : 1.0;  // else s9 is in qjk
  const size_t row = (size_t)i * a.N;
  if (lk) {
    atomicAdd(&a.S[row + k], sc * Sik);
    atomicAdd(&a.P[row + k], sc * Pik);
    if (PGRAD) {
      pg.s9 += Pik;
      pg.alp = fma(Wik, a.da1[(size_t)k * a.N + i], pg.alp);
      pg.a1 = fma(Wik, a.da1[row + k], pg.a1);
      pg.a2 = fma(Wik, a.da2[row + k], pg.a2);
    }
  }
  const int jt = j0 + GroupSum<J>::mine();
  if (GroupSum<J>::owner() && (!GUARD || (iok && jt > i))) {
    atomicAdd(&a.S[row + jt], sc * gS.a);
    atomicAdd(&a.P[row + jt], sc * gP.a);
    if (PGRAD) {
      pg.alp = fma(gW.a, a.da1[(size_t)jt * a.N + i], pg.alp);
      pg.a1 = fma(gW.a, a.da1[row + jt], pg.a1);
      pg.a2 = fma(gW.a, a.da2[row + jt], pg.a2);
    }
  }
}

}  // namespace

// A warp task is a tile of J consecutive middle atoms j, a chunk of eight
// outer atoms k > j and il consecutive inner atoms i < j: lane (q, l) takes
// k = kc + l, keeps the J (j, k) records and sums in registers, and walks
// every fourth i of the range (group q).  blockIdx = (tasks (tile, chunk) of
// the warps, i range, structure).  Eight middle atoms per lane keep one
// (i, k) reduction per eight triples; with parameter gradients (three sums
// per pair) four, which fit the registers.  Sums leave by FP64 reductions at
// L2, half a reduction per triple.
template <int J, bool GRAD, bool PGRAD>
__global__ void __launch_bounds__(128) atm_tiled64_kernel(Ctx c, int il) {
  const int b = blockIdx.z;
  const int n = c.w.n_eff[b];
  const int lane = threadIdx.x & 31;
  const int task = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  // groups of eight middle atoms, the top one n - 9 .. n - 2, so that all
  // chunks of outer atoms are full and what does not divide by eight is left to
  // the lowest group, which has the fewest inner atoms (its first j may be < 1)
  constexpr int R = A6_K / J;  // tiles per eight middle atoms
  const int NG = n < 3 ? 0 : (n - 2 + A6_K - 1) / A6_K;
  if (task >= R * (NG * (NG + 1) / 2)) return;
  const int sub = task % R, pt = task / R;
  int u = (int)((sqrtf(8.0f * (float)pt + 1.0f) - 1.0f) * 0.5f);
  while ((u + 1) * (u + 2) / 2 <= pt) ++u;
  while (u > 0 && u * (u + 1) / 2 > pt) --u;
  const int ch = pt - u * (u + 1) / 2;
  const int jg = n - 1 - A6_K * (u + 1), j0 = jg + J * sub;
  const int kc = jg + 1 + A6_K * ch;
  const int jend = j0 + J;
  if (jend < 2) return;
  const int ib0 = blockIdx.y * il;
  const int iend = min(ib0 + il, jend - 1);  // i < j <= jend - 1
  if (ib0 >= iend) return;
  const int N = c.N;
  const size_t base = (size_t)b * N * N;
  A6 a;
  a.T = c.w.pr4 + base;
  a.S = GRAD ? c.w.pr_S + base : nullptr;
  a.P = GRAD ? c.w.pr_P + base : nullptr;
  a.da1 = PGRAD ? c.w.pr_da1 + base : nullptr;
  a.da2 = PGRAD ? c.w.pr_da2 + base : nullptr;
  a.e3 = c.w.e3 + (size_t)b * N;
  a.cut2 = c.cut3_sq;
  a.alp6 = c.par.alp / 6.0;
  a.s9 = c.par.s9;
  a.n = n;
  a.N = N;
  const double *far2 = c.w.rowmax + (size_t)b * N;
  const int k = kc + (lane & 7);
  const bool kok = k < n;
  const double s9q = (PGRAD || !GRAD) ? 1.0 : a.s9;
  double zjk[J], ujk[J], tjk[J], qjk[J], Sjk[J], Pjk[J], Wjk[J];
  bool far = kok && far2[k] > a.cut2;
#pragma unroll
  for (int t = 0; t < J; ++t) {
    const int jt = j0 + t;
    PairRec r{0.0, 0.0, 0.0, 0.0};
    if (jt > 0 && kok && jt < k) r = a.T[(size_t)jt * N + k];
    zjk[t] = r.x;
    ujk[t] = r.u;
    tjk[t] = 6.0 * r.t;
    qjk[t] = s9q * r.q;  // 0 where (j, k) is not a pair: every product vanishes
    Sjk[t] = Pjk[t] = Wjk[t] = 0.0;
    far |= jt > 0 && far2[jt] > a.cut2;
  }
  const bool task_far = __any_sync(0xffffffffu, far);
  double Ek = 0.0;
  A6Pg pg;
  for (int ib = ib0; ib < iend; ib += 4) {
    const int i = ib + (lane >> 3);
    const bool iok = i < iend;
    const bool mask = task_far || __any_sync(0xffffffffu, iok && far2[i] > a.cut2);
    const bool guard = ib + 4 > iend || ib + 4 > j0;
    if (mask)
      a6_step<J, GRAD, PGRAD, true, true>(a, j0, k, kok, ib, i, iok, zjk, ujk, tjk, qjk, Sjk, Pjk,
                                          Wjk, Ek, pg);
    else if (guard)
      a6_step<J, GRAD, PGRAD, true, false>(a, j0, k, kok, ib, i, iok, zjk, ujk, tjk, qjk, Sjk, Pjk,
                                           Wjk, Ek, pg);
    else
      a6_step<J, GRAD, PGRAD, false, false>(a, j0, k, kok, ib, i, iok, zjk, ujk, tjk, qjk, Sjk,
                                            Pjk, Wjk, Ek, pg);
  }
  // the four groups' (j, k) sums: two exchanges leave each lane J / 4 of them
  const double sc = PGRAD ? a.s9 : 1.0;
  const int q = lane >> 3;
  if (GRAD) {
#pragma unroll
    for (int t = 0; t < J / 4; ++t) {
      const int jt = j0 + t + (J / 4) * q;  // bit 16 picks the upper half, bit 8 the quarter
      auto join = [&](const double (&v)[J]) {
        const double lo = lane_split(v[t], v[t + J / 2], 16);
        const double hi = lane_split(v[t + J / 4], v[t + J / 4 + J / 2], 16);
        return lane_split(lo, hi, 8);
      };
      const double sv = join(Sjk), pv = join(Pjk);
      const double wv = PGRAD ? join(Wjk) : 0.0;
      if (jt > 0 && kok && jt < k) {
        const size_t o = (size_t)jt * N + k;
        atomicAdd(&a.S[o], sc * sv);
        atomicAdd(&a.P[o], sc * pv);
        if (PGRAD) {
          pg.alp = fma(wv, a.da1[(size_t)k * N + jt], pg.alp);
          pg.a1 = fma(wv, a.da1[o], pg.a1);
          pg.a2 = fma(wv, a.da2[o], pg.a2);
        }
      }
    }
  } else {
    const double third = a.s9 / 3.0;
    Ek += __shfl_xor_sync(0xffffffffu, Ek, 8);
    Ek += __shfl_xor_sync(0xffffffffu, Ek, 16);
    if (q == 0 && kok && Ek != 0.0) atomicAdd(&a.e3[k], Ek * third);
#pragma unroll
    for (int t = 0; t < J; ++t) {
      const double ej = warp_sum(Pjk[t]);
      if (lane == 0 && j0 + t > 0 && ej != 0.0) atomicAdd(&a.e3[j0 + t], ej * third);
    }
  }
  if (PGRAD) {
    const double alp3 = c.par.alp / 3.0;
    pg.s9 = warp_sum(pg.s9);
    pg.alp = warp_sum(pg.alp);
    pg.a1 = warp_sum(pg.a1);
    pg.a2 = warp_sum(pg.a2);
    if (lane == 0) {
      double *o = c.w.pgrad + (size_t)b * D4_PARAM_GRAD_STRIDE;
      atomicAdd(&o[3], -a.s9 * alp3 * pg.a1);
      atomicAdd(&o[4], -a.s9 * alp3 * pg.a2);
      atomicAdd(&o[5], pg.s9);
      atomicAdd(&o[6], -a.s9 * (1.0 / 3.0) * pg.alp);
    }
  }
}

template <int J, bool GRAD, bool PGRAD>
static void launch_tiled64(const Ctx &c, cudaStream_t st) {
  const int N = c.N;
  if (N < 3) return;
  const long long NG = (N - 2 + A6_K - 1) / A6_K;
  const long long tasks = (A6_K / J) * NG * (NG + 1) / 2;
  // inner atoms per task: 32 (the ends of a task cost 1 % of eight steps, and
  // a task of 200 inner atoms alone on its SM would outlast the rest of a
  // batch), down to 8 where an SM would get fewer than 128 tasks (301 atoms
  // 564 -> 463 us, 360 x 30 271 -> 254), 4 where it would get fewer than 32
  // (57 atoms 30 -> 20; 360 x 30, which has more, loses by it: 325)
  int il = 32;
  auto count = [&]() { return tasks * c.B * ((N + il - 1) / il); };
  while (il > 8 && count() < 128LL * sm_count()) il >>= 1;
  if (count() < 32LL * sm_count()) il = 4;
  // one warp per CTA spreads few tasks over the SMs; four where there are many
  const int warps = count() < 64LL * sm_count() ? 1 : 4;
  const dim3 grid((unsigned)((tasks + warps - 1) / warps), (unsigned)((N + il - 1) / il),
                  (unsigned)c.B);
  atm_tiled64_kernel<J, GRAD, PGRAD><<<grid, 32 * warps, 0, st>>>(c, il);
}

void launch_atm_tiled64(const Ctx &c, cudaStream_t st) {
  if (c.flags & D4_FLAG_PARAM_GRAD)
    launch_tiled64<4, true, true>(c, st);
  else if (c.flags & D4_FLAG_GRADIENT)
    launch_tiled64<8, true, false>(c, st);
  else
    launch_tiled64<8, false, false>(c, st);
}

}  // namespace d4
