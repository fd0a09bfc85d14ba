// Register-tiled ATM of the precision form: all triples i < j < k of
// structures with unit energy weights (any size; padding atoms anywhere) that
// do not run over neighbour triples.  Energy weights run the per-triple kernel
// (d4_mixed.cu, atm_mixed_kernel).
//
// Bound by FP32 issue and latency (512 structures of 8..200 atoms: 0.70 of the
// issue slots at 16 warps per SM).  The
// pair sums leave by 8-byte reductions at L2 instead of shared-memory atomics
// (compare-and-swap loops), so no structure size is special and the sums of
// the parameter gradients fit beside them; the (i, j) sums cross lanes through
// shared memory (24 instructions per step; halving exchanges took 56).  Lanes
// holding 4 middle x 2 outer atoms (fewer exchanges, more tasks) were slower,
// 664 us, and so were direct loads instead of staged copies, 563.
// Measured, ATM stage, against a tile kernel with the sums in shared memory
// (N <= 234; no parameter gradients) and the per-triple kernel elsewhere: 512
// structures of 8..200 atoms 572 -> 481 us; 256 of 20..150 with parameter
// gradients 793 -> 245; 997 atoms 2115 -> 503; 1000 of 5..60, energies only,
// 110 -> 55.
#include "d4_atm.cuh"
#include "d4_common.cuh"
#include "d4_kernels.cuh"

namespace d4 {

namespace {

constexpr int A3_THREADS = 128;
constexpr int A3_ROW = 10;        // row and group strides of the (i, j) sums in shared memory
constexpr int A3_GROUP = 88;      // (float2; no bank conflicts)
constexpr int A3_STAGES = 3;      // staged chunks of eight inner atoms per warp
constexpr int A3_REC = 2 * A3 + 1;  // float4 per staged row: the four groups' broadcasts in
                                    // different banks

// Halving exchanges over the lane bits H, H/2, ... (STEPS of them): v[p]
// for p < NV >> STEPS ends as the sum over the 2^STEPS lanes that differ in
// those bits of the value with index p + (NV/2) bit(H) + (NV/4) bit(H/2) + ...
template <int NV, int H, int STEPS>
__device__ __forceinline__ void halving(float (&v)[NV]) {
  const int lane = threadIdx.x & 31;
#pragma unroll
  for (int s = 0; s < STEPS; ++s) {
    const int m = NV >> (s + 1), h = H >> s;
    const bool up = (lane & h) != 0;
#pragma unroll
    for (int q = 0; q < m; ++q) {
      const float keep = up ? v[q + m] : v[q];
      const float send = up ? v[q] : v[q + m];
      v[q] = keep + __shfl_xor_sync(0xffffffffu, send, h);
    }
  }
}

// 16 bytes of global memory to shared memory, or zeros.
__device__ __forceinline__ void copy16(float4 *dst, const float4 *src, bool ok) {
  const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
  asm volatile("cp.async.ca.shared.global [%0], [%1], 16, %2;" ::"r"(d), "l"(src),
               "r"(ok ? 16 : 0) : "memory");
}

struct A3Pair {
  const float4 *__restrict__ T;
  const float4 *__restrict__ Tda;  // PGRAD: (dlogR0/da1, dlogR0/da2, log(R0/r), -)
  float2 *SP;
  double *e3;
  double esc;  // factor of the energies added to e3 directly
  float cut2, alp3h;
  int N;
};

struct A3Pg {
  float s9 = 0.f, alp = 0.f, a1 = 0.f, a2 = 0.f;
  __device__ __forceinline__ void add(float w, const float4 &d) {
    a1 = fmaf(w, d.x, a1);
    a2 = fmaf(w, d.y, a2);
    alp = fmaf(w, d.z, alp);
  }
};

// One step: inner atom i of this lane's group against the eight middle atoms
// j0 .. j0 + 7 and the lane's outer atom k.  rec: the staged records (i, j) and
// (i, k) of the group's row, zeros where that is not a pair of the task (whose
// triples then vanish).  MASK: an atom of the step has a pair beyond the
// cutoff, so each triple takes its weight, (f_ij f_ik + f_ij f_jk + f_ik f_jk)
// / 3 (f: pair inside; 1, 1/3 or 0).  Of a 1/3 triple (weighted energy e_w)
// the atom of both inside pairs gets nothing and the other two e_w / 2 each
// (the reference's attribution): the row sums give the latter e_w / 6 through
// their inside pair and e_w / 3 through the outside one (atm_mirror_kernel),
// the former 2 e_w / 6, which leaves here as -e_w / 3 (Eik, Ek, s_cj).
template <bool GRAD, bool PGRAD, bool MASK>
__device__ __forceinline__ void a3_step(const A3Pair &a, const float4 *rec, int j0,
                                        unsigned jmask, int k, bool kok, int i, bool iok,
                                        const float (&zjk)[A3], const float (&izjk)[A3],
                                        const float (&ejk)[A3], const float (&qjk)[A3],
                                        float (&Sjk)[A3], float (&Pjk)[A3], float (&Wjk)[A3],
                                        float &Ek, float *s_cj, float2 *s_red, A3Pg &pg) {
  const int l = threadIdx.x & 7;
  const size_t row = (size_t)i * a.N;
  const float4 pik = rec[A3 + l];
  const float y = pik.x, iy38 = 0.375f * pik.y;
  const bool fik = !MASK || y <= a.cut2;
  float Sik = 0.f, Pik = 0.f, Wik = 0.f, Eik = 0.f, ei = 0.f;
  float wij[PGRAD ? A3 : 1];
  if (GRAD) __syncwarp();  // s_red: the last step's sums have been read
#pragma unroll
  for (int t = 0; t < A3; ++t) {
    const float4 pij = rec[t];
    const float x = pij.x, z = zjk[t];
    bool fij = true, fjk = true;
    int m = 3;
    float qij = pij.w;
    if (MASK) {
      fij = x <= a.cut2;
      fjk = z <= a.cut2;
      m = (int)fij + (int)fik + (int)fjk;
      if (GRAD) qij *= m == 3 ? 1.f : (m == 2 ? (1.0f / 3.0f) : 0.f);
      else qij = m >= 2 ? qij : 0.f;
    }
    // atm_triple (d4_atm.cuh) with its sums in place
    const float u = x - y, A = u + z, B = fmaf(2.0f, x, -A), C = z - u;
    const float AB = A * B, h = pij.y * (iy38 * izjk[t]);
    const float w = fmaf(AB * C, h, 1.0f);
    const float fd = sfu_rcp(fmaf(pij.z, pik.z * ejk[t], 1.0f));
    const float Q = qij * (pik.w * qjk[t]);
    const float cq = Q * fd;
    const float eu = cq * w;
    if (!GRAD) {
      // atom energies in units of eu / 3: all inside gives every atom 1, else
      // nothing to the atom of both inside pairs and 1/2 to the other two
      if (MASK && m == 2) {
        const float e2 = 0.5f * eu;
        ei += fjk ? e2 : 0.f;
        Eik += fij ? e2 : 0.f;  // (of atom k)
        Pjk[t] += fik ? e2 : 0.f;
      } else {
        ei += eu;
        Eik += eu;
        Pjk[t] += eu;
      }
      continue;
    }
    if (MASK) {  // energies of the 1/3 triples, for the atom of their inside pairs
      const float e2 = m == 2 ? eu : 0.f;
      ei += fjk ? 0.f : e2;
      Ek += fij ? 0.f : e2;
      if (!fik) s_cj[32 * t] += e2;
    }
    const float U = cq * h;
    const float V = fmaf(eu, fmaf(-a.alp3h, fd, a.alp3h - 2.5f), cq);
    const float sm = fmaf(A, C, AB), df = fmaf(-A, C, AB);
    Sik = fmaf(U, fmaf(-B, C, sm), fmaf(V, pik.y, Sik));
    Sjk[t] = fmaf(U, fmaf(B, C, df), fmaf(V, izjk[t], Sjk[t]));
    Pik += eu;
    Pjk[t] += eu;
    s_red[A3_ROW * t + l] = make_float2(fmaf(U, fmaf(B, C, -df), V * pij.y), eu);
    if (PGRAD) {
      const float wv = fmaf(-eu, fd, eu);
      Wik += wv;
      Wjk[t] += wv;
      wij[t] = wv;
    }
  }
  if (!GRAD || MASK) {  // energies of atom i over the group's lanes
    ei += __shfl_xor_sync(0xffffffffu, ei, 1);
    ei += __shfl_xor_sync(0xffffffffu, ei, 2);
    ei += __shfl_xor_sync(0xffffffffu, ei, 4);
    if (iok && l == 0 && ei != 0.f) atomicAdd(&a.e3[i], (double)ei * a.esc);
  }
  if (!GRAD) {
    Ek += Eik;
  } else {
    if (iok && kok && k > i) {
      red2(&a.SP[row + k], Sik, Pik);
      if (PGRAD) {
        pg.s9 += Pik;
        pg.add(Wik, a.Tda[row + k]);
      }
    }
    // the (i, j) sums over the eight lanes: lane l adds up row l of s_red
    __syncwarp();
    float s = 0.f, e = 0.f;
    const float4 *r4 = reinterpret_cast<const float4 *>(s_red + A3_ROW * l);
#pragma unroll
    for (int t = 0; t < A3 / 2; ++t) {
      const float4 r = r4[t];
      s += r.x + r.z;
      e += r.y + r.w;
    }
    const bool ok = iok && j0 + l > i && ((jmask >> l) & 1u);
    if (ok) red2(&a.SP[row + j0 + l], s, e);
    if (PGRAD) {
      float (&wv)[A3] = *reinterpret_cast<float(*)[A3]>(&wij[0]);
      halving<A3, 4, 3>(wv);  // lane l: value l
      if (ok) pg.add(wv[0], a.Tda[row + j0 + l]);
    }
  }
}

}  // namespace

// Running task counts of the structures in launch order (largest first),
// [0] = 0 .. [B], and the task counter behind them; in the room of dEdcn,
// which is written after the ATM.  One CTA.
__global__ void __launch_bounds__(1024) atm32_plan_kernel(Ctx c, int s) {
  __shared__ long long s_sum[32];
  long long *first = reinterpret_cast<long long *>(c.w.dEdcn);
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  long long base = 0;
  for (int b0 = 0; b0 < c.B; b0 += 1024) {
    long long v = 0;
    if (b0 + tid < c.B) {
      const int b = c.w.sorder[b0 + tid], n = c.w.n_eff[b];
      v = atm_sparse_mode(c, b, n) ? 0 : a3_tasks(n, s);
    }
    long long x = v;  // inclusive scan over the CTA
    for (int o = 1; o < 32; o <<= 1) {
      const long long y = __shfl_up_sync(0xffffffffu, x, o);
      if (lane >= o) x += y;
    }
    if (lane == 31) s_sum[warp] = x;
    __syncthreads();
    if (warp == 0) {
      long long y = s_sum[lane];
      for (int o = 1; o < 32; o <<= 1) {
        const long long z = __shfl_up_sync(0xffffffffu, y, o);
        if (lane >= o) y += z;
      }
      s_sum[lane] = y;
    }
    __syncthreads();
    x += base + (warp > 0 ? s_sum[warp - 1] : 0);
    if (b0 + tid < c.B) first[b0 + tid + 1] = x;
    base += s_sum[31];
    __syncthreads();
  }
  if (tid == 0) {
    first[0] = 0;
    first[c.B + 1] = 0;  // the task counter
  }
}

// A warp task is a tile of eight consecutive middle atoms j, eight outer atoms
// k > j and 8 s consecutive inner atoms i < j: lane (q, l) takes k = kc + l,
// keeps the eight (j, k) records and sums in registers and walks every fourth
// i of the range (group q).  The (i, j) and (i, k) records are copied to shared
// memory two chunks of eight i ahead.  Per i a lane evaluates eight triples
// from one (i, k) record and eight broadcast (i, j) records, adds its (i, k)
// sums with one reduction at L2, and the group's (i, j) sums change lanes
// through shared memory for another.  Warps take tasks from a counter, largest structures
// first.
template <bool GRAD, bool PGRAD>
__global__ void __launch_bounds__(A3_THREADS, PGRAD ? 3 : 4) atm32_kernel(Ctx c, int s) {
  __shared__ float s_c[A3_THREADS / 32][A3 * 32];
  __shared__ float4 s_rec[A3_THREADS / 32][A3_STAGES][8 * A3_REC];
  __shared__ __align__(16) float2 s_sum[A3_THREADS / 32][4 * A3_GROUP];
  const int lane = threadIdx.x & 31, q = lane >> 3;
  const int N = c.N;
  const long long *first = reinterpret_cast<const long long *>(c.w.dEdcn);
  unsigned long long *next =
      reinterpret_cast<unsigned long long *>(c.w.dEdcn) + c.B + 1;
  const long long total = first[c.B];
  auto take = [&]() {
    unsigned long long t = 0;
    if (lane == 0) t = atomicAdd(next, 1ull);
    return (long long)__shfl_sync(0xffffffffu, t, 0);
  };
  int at = 0;  // position in launch order of the last task's structure
  for (long long task = take(); task < total;) {
    const long long following = take();  // on its way while this task runs
    // the structure: tasks come in order, so search on from the last one
    if (task >= first[at + 1]) {
      int lo = at + 1, hi = c.B - 1;
      while (lo < hi) {
        const int mid = (lo + hi) >> 1;
        if (task >= first[mid + 1])
          lo = mid + 1;
        else
          hi = mid;
      }
      at = lo;
    }
    const int b = c.w.sorder[at];
    const int n = c.w.n_eff[b];
    // tile, chunk and inner range
    const A3Task at3 = a3_task(task - first[at], n, s);
    const int j0 = n - 1 - A3 * (at3.u + 1), kc = j0 + 1 + A3 * at3.ch, jend = j0 + A3;
    const int ib0 = at3.ip * A3 * s, iend = min(ib0 + A3 * s, jend - 1);
    const size_t bN = (size_t)b * N;
    A3Pair a;
    a.T = c.w.ptf + bN * N;
    a.Tda = PGRAD ? c.w.ptf_da + bN * N : nullptr;
    a.SP = GRAD ? c.w.prSP32 + bN * N : nullptr;
    a.e3 = c.w.e3 + bN;
    a.esc = GRAD ? (PGRAD ? c.par.s9 : 1.0) * (-1.0 / 3.0) : c.par.s9 / 3.0;
    a.cut2 = c.pf.cut3 * c.pf.cut3;
    a.alp3h = 0.5f * c.pf.alp3;
    a.N = N;
    const bool gaps = c.w.n_real[b] != n;
    const int *Z = c.w.z + bN;
    const float *far2 = reinterpret_cast<const float *>(c.w.atm_rowmax) + bN;
    const int k = kc + (lane & 7);
    const bool kok = k < n && (!gaps || Z[k] != 0);
    // s9 goes into the (j, k) records; parameter gradients and energies
    // without gradient apply it at the end
    const float s9q = (GRAD && !PGRAD) ? c.pf.s9 : 1.f;
    float zjk[A3], izjk[A3], ejk[A3], qjk[A3], Sjk[A3], Pjk[A3], Wjk[A3];
    unsigned jmask = 0u;
    bool far = kok && far2[k] > a.cut2, task_far = false;
#pragma unroll
    for (int tt = 0; tt < A3; ++tt) {
      const int jt = j0 + tt;
      const bool jok = jt > 0 && (!gaps || Z[jt] != 0);
      jmask |= (unsigned)jok << tt;
      float4 r = make_float4(0.f, 0.f, 0.f, 0.f);
      if (kok && jok && jt < k) r = a.T[(size_t)jt * N + k];
      zjk[tt] = r.x;
      izjk[tt] = r.y;
      ejk[tt] = 6.0f * r.z;  // prescaled for atm_triple<., true>
      qjk[tt] = s9q * r.w;   // 0 where (j, k) is not a pair: every product vanishes
      Sjk[tt] = Pjk[tt] = Wjk[tt] = 0.f;
      far |= jok && far2[jt] > a.cut2;
      task_far |= r.x > a.cut2;
    }
    task_far = __any_sync(0xffffffffu, task_far);  // a (j, k) beyond the cutoff
    for (int ib = ib0 + lane; ib < iend; ib += 32) far |= far2[ib] > a.cut2;
    const bool any_far = __any_sync(0xffffffffu, far);
    float Ek = 0.f;
    float *cj = s_c[threadIdx.x >> 5] + lane;
    if (GRAD && any_far) {
#pragma unroll
      for (int tt = 0; tt < A3; ++tt) cj[32 * tt] = 0.f;
    }
    A3Pg pg;
    // records of eight inner atoms at a time: entry t of row r is (i, j0 + t),
    // 8 + t (i, kc + t), i = first + r; copied two chunks ahead
    float4(*stage)[8 * A3_REC] = s_rec[threadIdx.x >> 5];
    float2 *red = s_sum[threadIdx.x >> 5] + A3_GROUP * q;
    auto fetch = [&](int first_i, int st) {
      if (first_i < iend) {
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const int slot = lane + 32 * e, r = slot >> 4, col = slot & 15;
          const int i = first_i + r, x = col < A3 ? j0 + col : kc + col - A3;
          const bool ok = i < iend && x > i && (col < A3 ? ((jmask >> col) & 1u) != 0u : x < n) &&
                          (!gaps || (Z[i] != 0 && Z[x] != 0));
          copy16(&stage[st][A3_REC * r + col], a.T + (ok ? (size_t)i * N + x : 0), ok);
        }
      }
      asm volatile("cp.async.commit_group;" ::: "memory");
    };
    __syncwarp();  // every lane is done with the last task's records
    fetch(ib0, 0);
    fetch(ib0 + 8, 1);
    int st = 0;
    for (int ib = ib0; ib < iend; ib += 8) {
      fetch(ib + 16, st >= A3_STAGES - 2 ? st - (A3_STAGES - 2) : st + 2);
      asm volatile("cp.async.wait_group 2;" ::: "memory");
      __syncwarp();
#pragma unroll 1
      for (int half = 0; half < 2; ++half) {
        const int i = ib + 4 * half + q;
        if (ib + 4 * half >= iend) break;
        const bool iok = i < iend && (!gaps || Z[i] != 0);
        const float4 *rec = stage[st] + A3_REC * (4 * half + q);
        // a pair of the step beyond the cutoff (any_far: an atom of the task has one;
        // by atoms alone nearly all steps of 997 atoms took their masks)
        const bool mask = any_far && (task_far || __any_sync(0xffffffffu,
                                                             rec[lane & 7].x > a.cut2 ||
                                                                 rec[A3 + (lane & 7)].x > a.cut2));
        if (mask)
          a3_step<GRAD, PGRAD, true>(a, rec, j0, jmask, k, kok, i, iok, zjk, izjk, ejk, qjk, Sjk,
                                     Pjk, Wjk, Ek, cj, red, pg);
        else
          a3_step<GRAD, PGRAD, false>(a, rec, j0, jmask, k, kok, i, iok, zjk, izjk, ejk, qjk, Sjk,
                                      Pjk, Wjk, Ek, cj, red, pg);
      }
      __syncwarp();
      if (++st == A3_STAGES) st = 0;
    }
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    // the four groups' (j, k) sums: two exchanges leave group q the pairs of
    // middle atoms 2 q and 2 q + 1
    constexpr int K = GRAD ? (PGRAD ? 3 : 2) : 1, NV = K * A3;
    float v[NV];
#pragma unroll
    for (int tt = 0; tt < A3; ++tt) {
      if (GRAD) {
        v[tt * K] = Sjk[tt];
        v[tt * K + 1] = Pjk[tt];
        if (PGRAD) v[tt * K + K - 1] = Wjk[tt];
      } else {
        v[tt] = Pjk[tt];
      }
    }
    halving<NV, 16, 2>(v);
    if (GRAD) {
      if (any_far) {  // the 1/3 triples' common middle and outer atoms
#pragma unroll
        for (int tt = 0; tt < A3; ++tt) {
          const float e = warp_sumf(cj[32 * tt]);
          if (lane == 0 && ((jmask >> tt) & 1u) && e != 0.f)
            atomicAdd(&a.e3[j0 + tt], (double)e * a.esc);
        }
        Ek += __shfl_xor_sync(0xffffffffu, Ek, 8);
        Ek += __shfl_xor_sync(0xffffffffu, Ek, 16);
        if (q == 0 && kok && Ek != 0.f) atomicAdd(&a.e3[k], (double)Ek * a.esc);
      }
#pragma unroll
      for (int p = 0; p < 2; ++p) {
        const int jt = j0 + 2 * q + p;
        if (kok && jt < k && ((jmask >> (2 * q + p)) & 1u)) {
          red2(&a.SP[(size_t)jt * N + k], v[p * K], v[p * K + 1]);
          if (PGRAD) pg.add(v[p * K + K - 1], a.Tda[(size_t)jt * N + k]);
        }
      }
    } else {
      // energies: of the middle atoms over the outer ones, of the outer atoms
#pragma unroll
      for (int p = 0; p < 2; ++p) {
        float ej = v[p];
        ej += __shfl_xor_sync(0xffffffffu, ej, 1);
        ej += __shfl_xor_sync(0xffffffffu, ej, 2);
        ej += __shfl_xor_sync(0xffffffffu, ej, 4);
        if ((lane & 7) == 0 && ((jmask >> (2 * q + p)) & 1u) && ej != 0.f)
          atomicAdd(&a.e3[j0 + 2 * q + p], (double)ej * a.esc);
      }
      Ek += __shfl_xor_sync(0xffffffffu, Ek, 8);
      Ek += __shfl_xor_sync(0xffffffffu, Ek, 16);
      if (q == 0 && kok && Ek != 0.f) atomicAdd(&a.e3[k], (double)Ek * a.esc);
    }
    if (PGRAD) {
      pg.s9 = warp_sumf(pg.s9);
      pg.alp = warp_sumf(pg.alp);
      pg.a1 = warp_sumf(pg.a1);
      pg.a2 = warp_sumf(pg.a2);
      if (lane == 0) {  // d fd / d(alp/3 sum log(R0/r)) = -fd (1 - fd)
        double *o = c.w.pgrad + (size_t)b * D4_PARAM_GRAD_STRIDE;
        const double s9 = c.par.s9, w = -s9 * (c.par.alp / 3.0);
        atomicAdd(&o[3], w * (double)pg.a1);
        atomicAdd(&o[4], w * (double)pg.a2);
        atomicAdd(&o[5], (double)pg.s9);
        atomicAdd(&o[6], -s9 * (1.0 / 3.0) * (double)pg.alp);
      }
    }
    task = following;
  }
}

// ATM over the neighbour triples of structures in sparse mode (atm_sparse_mode;
// unit energy weights): a CTA per centre atom j, whose neighbours L (ascending;
// runs of consecutive atoms where the structure is in spatial order) form the
// triples (i, j, k), i < k, with r_ij and r_jk inside the cutoff.  A triple
// with r_ik outside has no other centre; one with all sides inside is taken at
// its smallest atom (j < i).  A warp task is 32 neighbours k, a lane each with
// its (j, k) record and sums in registers, against up to 64 neighbours i, four
// rows' (i, k) records in flight: the (i, k) sums leave by one reduction at L2
// each, the (i, j) sums of four rows cross lanes by halving exchanges (9 shuffles;
// through shared memory they took 22 of its wavefronts and those bound the kernel at
// 0.80 of their rate; now it is issue, 0.80: 16000 atoms, cutoff 25 Bohr, 8.0 -> 7.1
// ms).  Atom
// energies come from the pair sums (atm_mirror_kernel); only the energies e_w
// of the centre's 1/3 triples, which it gets nothing of, leave here as -e_w /
// 3 (see a3_step).  Energies without gradient have no pair sums and add up
// atom energies instead, in units of eu / 6.
constexpr int SP_THREADS = 512, SP_ROWS = 4, SP_BLOCK = 64;

// Tasks of the first m chunks: chunk ec has ec / 2 + 1 blocks of rows.
__device__ __forceinline__ int sp_tasks(int m) { return (m + 1) * (m + 1) / 4; }

template <bool GRAD, bool PGRAD>
__global__ void __launch_bounds__(SP_THREADS, 2) atm_sparse32_kernel(Ctx c) {
  extern __shared__ float4 s_rec[];  // [ATM_SPARSE_DMAX] records (j, L[t])
  float2 *s_SP = reinterpret_cast<float2 *>(s_rec + ATM_SPARSE_DMAX);  // their sums
  int *s_L = reinterpret_cast<int *>(s_SP + ATM_SPARSE_DMAX);
  float *s_W = reinterpret_cast<float *>(s_L + ATM_SPARSE_DMAX);  // PGRAD: damping sums
  __shared__ float s_red[SP_THREADS / 32];
  __shared__ int s_next;
  const int b = blockIdx.y, N = c.N, n = c.w.n_eff[b];
  if ((int)blockIdx.x >= n || n < 3 || !atm_sparse_mode(c, b, n)) return;
  const size_t bN = (size_t)b * N;
  const int j = c.zsorted ? (int)blockIdx.x : c.w.atm_order[bN + blockIdx.x];
  if (c.w.z[bN + j] == 0) return;
  const int d = c.w.nbr_deg[bN + j];  // <= ATM_SPARSE_DMAX in sparse mode
  if (d < 2) return;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const float4 *T = c.w.ptf + bN * N;
  const float4 *Tda = PGRAD ? c.w.ptf_da + bN * N : nullptr;
  float2 *SP = GRAD ? c.w.prSP32 + bN * N : nullptr;
  const int *L = c.w.nbr + (bN + j) * N;
  for (int t = tid; t < d; t += SP_THREADS) {
    const int k = L[t];
    s_L[t] = k;
    s_rec[t] = T[(size_t)j * N + k];
    s_SP[t] = make_float2(0.f, 0.f);
    if (PGRAD) s_W[t] = 0.f;
  }
  if (tid == 0) s_next = SP_THREADS / 32;
  __syncthreads();
  const float cut2 = c.pf.cut3 * c.pf.cut3, alp3h = 0.5f * c.pf.alp3;
  const float s9 = (GRAD && !PGRAD) ? c.pf.s9 : 1.f;  // PGRAD, energies: at the end
  float Cj = 0.f;
  A3Pg pg;
  const int nch = (d + 31) / 32, tasks = sp_tasks(nch);
  for (int task = warp; task < tasks;) {
    // chunk ec of 32 neighbours k has ec / 2 + 1 blocks of 64 rows i
    int ec = (int)(2.0f * sqrtf((float)task));
    while (sp_tasks(ec + 1) <= task) ++ec;
    while (ec > 0 && sp_tasks(ec) > task) --ec;
    const int a_beg = SP_BLOCK * (task - sp_tasks(ec));
    const int a_end = min(min(a_beg + SP_BLOCK, d - 1), 32 * ec + 31);  // rows a < e
    const int e = 32 * ec + lane;
    const bool eok = e < d;
    const int k = eok ? s_L[e] : 0;
    const float4 pjk = eok ? s_rec[e] : make_float4(0.f, 0.f, 0.f, 0.f);
    const float z = pjk.x, ejk = 6.0f * pjk.z, qjk = s9 * pjk.w;
    float Sjk = 0.f, Pjk = 0.f, Wjk = 0.f;
    for (int a0 = a_beg; a0 < a_end; a0 += SP_ROWS) {
      float4 pik[SP_ROWS];
#pragma unroll
      for (int r = 0; r < SP_ROWS; ++r) {
        const int a = a0 + r;
        const bool ok = a < a_end && eok && e > a;
        pik[r] = ok ? T[(size_t)s_L[ok ? a : 0] * N + k] : make_float4(0.f, 0.f, 0.f, 0.f);
      }
      float wij[PGRAD ? SP_ROWS : 1];
      float v[GRAD ? 2 * SP_ROWS : SP_ROWS];  // the rows' sums (S, P), or energies
#pragma unroll
      for (int r = 0; r < SP_ROWS; ++r) {
        const int a = a0 + r;
        const int i = s_L[a < a_end ? a : 0];
        const bool in = pik[r].x <= cut2;
        const bool use = a < a_end && eok && e > a && (j < i || !in);
        float2 out = make_float2(0.f, 0.f);
        float wv = 0.f;
        if (__any_sync(0xffffffffu, use)) {
          // atm_triple (d4_atm.cuh) with its sums in place
          const float4 pij = s_rec[a];
          const float x = pij.x, y = pik[r].x;
          const float u = x - y, A = u + z, B = fmaf(2.0f, x, -A), C = z - u;
          const float AB = A * B, h = pij.y * (0.375f * pik[r].y * pjk.y);
          const float w = fmaf(AB * C, h, 1.0f);
          const float fd = sfu_rcp(fmaf(pij.z, pik[r].z * ejk, 1.0f));
          float qij = use ? pij.w : 0.f;
          if (GRAD && !in) qij *= 1.0f / 3.0f;
          const float Q = qij * (pik[r].w * qjk);
          const float cq = Q * fd, eu = cq * w;
          if (GRAD) {
            const float U = cq * h;
            const float V = fmaf(eu, fmaf(-alp3h, fd, alp3h - 2.5f), cq);
            const float sm = fmaf(A, C, AB), df = fmaf(-A, C, AB);
            out = make_float2(fmaf(U, fmaf(B, C, -df), V * pij.y), eu);
            Sjk = fmaf(U, fmaf(B, C, df), fmaf(V, pjk.y, Sjk));
            Pjk += eu;
            Cj += in ? 0.f : eu;
            if (use)
              red2(&SP[(size_t)i * N + k], fmaf(U, fmaf(-B, C, sm), V * pik[r].y), eu);
            if (PGRAD) {
              wv = fmaf(-eu, fd, eu);
              Wjk += wv;
              pg.s9 += eu;
              if (use) pg.add(wv, Tda[(size_t)i * N + k]);
            }
          } else {
            // all sides inside: a third to each atom; else half to i and to k
            out.x = in ? 2.0f * eu : eu;
            Pjk += out.x;
            Cj += in ? 2.0f * eu : 0.f;
          }
        }
        if (GRAD) {
          v[2 * r] = out.x;
          v[2 * r + 1] = out.y;
        } else {
          v[r] = out.x;
        }
        if (PGRAD) wij[r] = wv;
      }
      // (i, j) sums: halving exchanges leave value lane >> 2 (2 r + component of
      // row r; energies lane >> 3, row r) to the lanes of a group
      float sum;
      if (GRAD) {
        float (&v8)[8] = *reinterpret_cast<float(*)[8]>(&v[0]);
        halving<8, 16, 3>(v8);
        sum = v8[0];
      } else {
        float (&v4)[4] = *reinterpret_cast<float(*)[4]>(&v[0]);
        halving<4, 16, 2>(v4);
        sum = v4[0] + __shfl_xor_sync(0xffffffffu, v4[0], 4);
      }
      sum += __shfl_xor_sync(0xffffffffu, sum, 2);
      sum += __shfl_xor_sync(0xffffffffu, sum, 1);
      {
        const int row = a0 + (lane >> 3), comp = GRAD ? (lane >> 2) & 1 : 0;
        if ((lane & (GRAD ? 3 : 7)) == 0 && row < a_end && sum != 0.f)
          atomicAdd(comp ? &s_SP[row].y : &s_SP[row].x, sum);
      }
      if (PGRAD) {
#pragma unroll
        for (int r = 0; r < SP_ROWS; ++r) {
          const float wv = warp_sumf(wij[r]);
          if (lane == 0 && wv != 0.f) atomicAdd(&s_W[a0 + r], wv);
        }
      }
    }
    if (eok) {
      if (GRAD && Sjk != 0.f) atomicAdd(&s_SP[e].x, Sjk);
      if (Pjk != 0.f) atomicAdd(GRAD ? &s_SP[e].y : &s_SP[e].x, Pjk);
      if (PGRAD && Wjk != 0.f) atomicAdd(&s_W[e], Wjk);
    }
    int nx = 0;
    if (lane == 0) nx = atomicAdd(&s_next, 1);
    task = __shfl_sync(0xffffffffu, nx, 0);
  }
  Cj = warp_sumf(Cj);
  if (lane == 0) s_red[warp] = Cj;
  __syncthreads();
  double *e3 = c.w.e3 + bN;
  if (tid == 0) {
    float t = 0.f;
    for (int w = 0; w < SP_THREADS / 32; ++w) t += s_red[w];
    const double f = GRAD ? (PGRAD ? c.par.s9 : 1.0) * (-1.0 / 3.0) : c.par.s9 / 6.0;
    if (t != 0.f) atomicAdd(&e3[j], (double)t * f);
  }
  for (int t = tid; t < d; t += SP_THREADS) {
    const int k = s_L[t];
    const float2 v = s_SP[t];
    if (GRAD) {
      if (v.x != 0.f || v.y != 0.f)
        red2(&SP[j < k ? (size_t)j * N + k : (size_t)k * N + j], v.x, v.y);
      if (PGRAD) pg.add(s_W[t], Tda[(size_t)j * N + k]);
    } else if (v.x != 0.f) {
      atomicAdd(&e3[k], (double)v.x * (c.par.s9 / 6.0));
    }
  }
  if (PGRAD) {  // d fd / d(alp/3 sum log(R0/r)) = -fd (1 - fd)
    pg.s9 = warp_sumf(pg.s9);
    pg.alp = warp_sumf(pg.alp);
    pg.a1 = warp_sumf(pg.a1);
    pg.a2 = warp_sumf(pg.a2);
    if (lane == 0) {
      double *o = c.w.pgrad + (size_t)b * D4_PARAM_GRAD_STRIDE;
      const double s9d = c.par.s9, w = -s9d * (c.par.alp / 3.0);
      atomicAdd(&o[3], w * (double)pg.a1);
      atomicAdd(&o[4], w * (double)pg.a2);
      atomicAdd(&o[5], (double)pg.s9);
      atomicAdd(&o[6], -s9d * (1.0 / 3.0) * (double)pg.alp);
    }
  }
}

// The lower half of the ATM pair sums from the upper one, 32 x 32 tiles through
// shared memory.  After the unit-weight kernels also the atom energies from the row sums
// (every triple reaches an atom through two of its pairs, a third of its
// energy each; a pair beyond the cutoff counts twice, see a3_step) and, with
// parameter gradients, the factor s9.  Bound by latency: loads carry no condition and a
// warp's eight sums leave by one exchange (512 structures of 8..200 atoms 42 -> 23 us;
// 16000 atoms 496 -> 335 us).
__global__ void __launch_bounds__(256) atm_mirror_kernel(Ctx c, bool rows, float s9) {
  __shared__ float2 s_t[32][33];
  __shared__ float s_e[32][33];
  __shared__ float s_sum[64];
  const int b = blockIdx.y, N = c.N, n = c.w.n_eff[b];
  int ti, tj;  // rows ti, columns tj >= ti
  tri_entry(blockIdx.x, tj, ti);
  if (tj * 32 >= n) return;
  // the sides of a triple with weight are within twice the cutoff
  if (c.far_skip && block_gap_sq(c, b, ti, tj) > 4.f * c.pf.cut3 * c.pf.cut3) return;
  float2 *SP = c.w.prSP32 + (size_t)b * N * N;
  double *e3 = c.w.e3 + (size_t)b * N;
  const float cut2 = c.pf.cut3 * c.pf.cut3;
  const float *far2 = reinterpret_cast<const float *>(c.w.atm_rowmax) + (size_t)b * N;
  const float4 *T = c.w.ptf + (size_t)b * N * N;
  const int *Z = c.w.z + (size_t)b * N;
  const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
  const int jr = tj * 32 + tx, jc = min(jr, N - 1);
  float2 v[4];
  int zi[4];
#pragma unroll
  for (int q = 0; q < 4; ++q) {  // (unconditional, so that all loads are in flight)
    const int i = ti * 32 + ty + 8 * q, ic = min(i, N - 1);
    zi[q] = Z[ic];
    v[q] = SP[(size_t)ic * N + jc];
  }
  const bool jok = jr < n && Z[jc] != 0;
  const bool far_j = rows && jok && far2[jc] > cut2;
  float e[8];  // row sums' terms, then those of the mirrored rows
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    const int r = ty + 8 * q, i = ti * 32 + r;
    const bool ok = jok && jr > i && zi[q] != 0;  // (i < jr < n)
    if (!ok) v[q] = make_float2(0.f, 0.f);
    if (ok && s9 != 1.f) {
      v[q].x *= s9;
      v[q].y *= s9;
      SP[(size_t)i * N + jr] = v[q];
    }
    e[q] = v[q].y;
    if (far_j && e[q] != 0.f && T[(size_t)i * N + jr].x > cut2) e[q] += e[q];
    s_t[r][tx] = v[q];
    if (rows) s_e[r][tx] = e[q];
  }
  __syncthreads();
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    const int r = ty + 8 * q;
    const int i = tj * 32 + r, j = ti * 32 + tx;  // destination (i > j)
    if (i < n && j < n && i > j) SP[(size_t)i * N + j] = s_t[tx][r];
    if (rows) e[4 + q] = s_e[tx][r];
  }
  if (rows) {
    halving<8, 16, 3>(e);
    e[0] += __shfl_xor_sync(0xffffffffu, e[0], 2);
    e[0] += __shfl_xor_sync(0xffffffffu, e[0], 1);
    const int q = tx >> 2;  // the sum that the lane ends with: bits 16, 8, 4
    if ((tx & 3) == 0) s_sum[(q < 4 ? 0 : 32) + ty + 8 * (q & 3)] = e[0];
    __syncthreads();
    if (threadIdx.x < 64) {  // (FP64 instructions of two warps, not eight)
      const float es = s_sum[threadIdx.x];
      if (es != 0.f)
        atomicAdd(&e3[(threadIdx.x < 32 ? ti : tj) * 32 + tx], (double)es * (1.0 / 6.0));
    }
  }
}

void launch_atm_mirror(const Ctx &c, cudaStream_t st, bool rows, float s9) {
  const unsigned T = (unsigned)(c.N + 31) / 32;
  atm_mirror_kernel<<<dim3(T * (T + 1) / 2, c.B), 256, 0, st>>>(c, rows, s9);
}

template <bool GRAD, bool PGRAD>
static void launch_sparse32(const Ctx &c, cudaStream_t st) {
  const int bytes = ATM_SPARSE_DMAX * (16 + 8 + 4 + (PGRAD ? 4 : 0));
  ensure_smem(atm_sparse32_kernel<GRAD, PGRAD>, bytes);
  atm_sparse32_kernel<GRAD, PGRAD><<<dim3(c.N, c.B), SP_THREADS, bytes, st>>>(c);
}

void launch_atm_sparse32(const Ctx &c, cudaStream_t st) {
  if (c.flags & D4_FLAG_PARAM_GRAD)
    launch_sparse32<true, true>(c, st);
  else if (c.flags & D4_FLAG_GRADIENT)
    launch_sparse32<true, false>(c, st);
  else
    launch_sparse32<false, false>(c, st);
}

void launch_atm32(const Ctx &c, cudaStream_t st) {
  if (c.N < 3) return;
  const int nsm = sm_count();
  const bool grad = (c.flags & D4_FLAG_GRADIENT) != 0;
  const bool pgrad = (c.flags & D4_FLAG_PARAM_GRAD) != 0;
  // inner atoms per task: 128 (finding, loading and flushing a task takes as
  // long as 1.5 of its steps: 8-atom steps 16 against 4 per task 559 to 652 us
  // for 512 structures of 8..200 atoms), fewer where a wave of warps would not
  // get two such tasks each
  const double triples = (double)c.B * c.N * c.N * c.N / 6.0;
  int s = 16;
  while (s > 1 && triples < 2.0 * 64 * 8 * s * 16.0 * nsm) s >>= 1;
  atm32_plan_kernel<<<1, 1024, 0, st>>>(c, s);
  const unsigned grid = (unsigned)((pgrad ? 3 : 4) * nsm);
  if (pgrad)
    atm32_kernel<true, true><<<grid, A3_THREADS, 0, st>>>(c, s);
  else if (grad)
    atm32_kernel<true, false><<<grid, A3_THREADS, 0, st>>>(c, s);
  else
    atm32_kernel<false, false><<<grid, A3_THREADS, 0, st>>>(c, s);
}

}  // namespace d4

extern "C" int64_t d4_selftest_atm_task(int32_t n, int32_t s, int64_t task, int32_t *out) {
  if (n < 3 || s < 1 || !out) return -1;
  const long long total = d4::a3_tasks(n, s);
  if (task < 0 || task >= total) return total;
  const d4::A3Task t = d4::a3_task(task, n, s);
  out[0] = t.ip;
  out[1] = t.u;
  out[2] = t.ch;
  return total;
}
