// The ATM triple of the precision form, shared by its ATM kernels
// (d4_mixed.cu, d4_atm32.cu).
#pragma once

#include "d4_common.cuh"

namespace d4 {

// 1 / x to the SFU's ~1 ulp (x >= 1 here: the ATM damping)
__device__ __forceinline__ float sfu_rcp(float x) {
  float y;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

// Adds (S, P) to a pair's sums, one 8-byte reduction at L2.
__device__ __forceinline__ void red2(float2 *p, float s, float e) {
  asm volatile("red.global.add.v2.f32 [%0], {%1, %2};" ::"l"(p), "f"(s), "f"(e) : "memory");
}

// ATM triple (i, j, k) of the precision form from its three pair records
// (r^2, 1/r^2, (R0/r)^(alp/3), sqrt(C6(q=0)) / r^3) of the pairs ij, ik,
// jk (x, y, z = their r^2).  With R = r_ij r_ik r_jk, the angular factor is
// w / R^3, w = 1 + 3/8 (x - y + z)(x + y - z)(y + z - x) / R^2, and C9 / R^3
// is the product Q of the records' fourth entries, so the energy without s9
// is eu = Q fd w with fd = 1 / (1 + 6 prod (R0/r)^(alp/3)) (the reference's
// damping, model/d4.py three-body term through damping/atm.py).  dex, dey,
// dez: d eu / d(x, y, z); qwg = Q w fd (1 - fd), for the parameter gradients.
struct AtmTri {
  float eu, dex, dey, dez, qwg;
};

// EZ6: ez arrives multiplied by 6 (a caller that holds the (j, k) record for
// many triples scales it once).
template <bool GRAD, bool EZ6 = false>
__device__ __forceinline__ AtmTri atm_triple(float x, float ix2, float ex, float qx, float y,
                                             float iy2, float ey, float qy, float z, float iz2,
                                             float ez, float qz, float alp3h) {
  AtmTri r;
  const float ir2 = ix2 * (iy2 * iz2);
  const float h = 0.375f * ir2;
  const float u = x - y;
  const float A = u + z, Bv = (x + y) - z, Cv = z - u;
  const float AB = A * Bv;
  const float w = fmaf(AB * Cv, h, 1.0f);
  // (rounding 1 + 6 prod drops its small values at distant triples alike;
  // measured on 16000 atoms the three-body energy stays within 1e-8 Eh of
  // the FP64 reference, and a Newton-corrected fd costs 3 % of the kernel)
  const float fd = EZ6 ? sfu_rcp(fmaf(ex, ey * ez, 1.0f))
                      : sfu_rcp(fmaf(6.0f, ex * (ey * ez), 1.0f));
  const float Q = qx * (qy * qz);
  const float cq = Q * fd;
  r.eu = cq * w;
  if (GRAD) {
    // U = 3/8 C9 fd / R^5, V = C9 / (2 R^3) (fd (2 - 5 w) + w alp/3 fd (1 - fd))
    //   = C9 fd / R^3 (1 + w (alp/6 (1 - fd) - 5/2))
    const float U = cq * h;
    const float V = cq * fmaf(w, fmaf(-alp3h, fd, alp3h - 2.5f), 1.0f);
    const float AC = A * Cv, BC = Bv * Cv;
    const float Sg = AB + AC + BC;
    r.dex = fmaf(U, fmaf(-2.0f, AB, Sg), V * ix2);
    r.dey = fmaf(U, fmaf(-2.0f, BC, Sg), V * iy2);
    r.dez = fmaf(U, fmaf(-2.0f, AC, Sg), V * iz2);
    r.qwg = Q * w * fmaf(-fd, fd, fd);
  } else {
    r.dex = r.dey = r.dez = r.qwg = 0.f;
  }
  return r;
}

// Whether the ATM of structure b runs over neighbour triples (centre-atom
// enumeration, atm_sparse_kernel) instead of all triples i < j < k: when
// every centre's neighbour list fits the kernel's shared memory and the
// centre-pair visits, sum_j deg_j (deg_j - 1) / 2, are fewer than half the
// n (n - 1) (n - 2) / 6 triples.  Counts come from atm_nbr_kernel; only
// structures of the global-accumulation path (N > 234) have them.
__device__ __forceinline__ bool atm_sparse_mode(const Ctx &c, int b, int n) {
  if (c.w.atm_cnt == nullptr) return false;
  const unsigned long long visits = c.w.atm_cnt[2 * b], dmax = c.w.atm_cnt[2 * b + 1];
  const unsigned long long nn = (unsigned long long)n;
  const unsigned long long all = nn * (nn - 1) * (nn - 2) / 6;
  return dmax <= (unsigned long long)ATM_SPARSE_DMAX && 2 * visits < all;
}

// ---------------------------------------------------------------- tasks of atm32_kernel

constexpr int A3 = 8;  // middle atoms per lane, and outer atoms per task

// Number of tasks of a structure of n atoms whose tasks cover 8 s inner atoms
// each.  Tiles of middle atoms are counted from the last (n - 9 .. n - 2), so
// that all chunks of outer atoms are full and the lowest tile, with the fewest
// inner atoms, takes what does not divide by eight (its first j may be < 1).
// Tile g from below has NG - g chunks of outer atoms and g / s + 1 ranges of
// inner atoms.
__host__ __device__ inline long long a3_tasks(int n, int s) {
  const long long ng = n < 3 ? 0 : (n - 2 + A3 - 1) / A3;
  long long t = 0;
  for (long long m = ng; m > 0; m -= s) t += m * (m + 1) / 2;
  return t;
}

// Task t of them: the inner range ip, tile u (from the top) and chunk ch of
// outer atoms.  (All of it in 64 bits: 47300 atoms have 2^31 tasks.)
struct A3Task {
  int ip, u, ch;
};
__host__ __device__ inline A3Task a3_task(long long t, int n, int s) {
  A3Task r;
  r.ip = 0;
  long long m = (n - 2 + A3 - 1) / A3;
  while (t >= m * (m + 1) / 2) {
    t -= m * (m + 1) / 2;
    m -= s;
    ++r.ip;
  }
  tri_entry(t, r.u, r.ch);
  return r;
}

}  // namespace d4
