// Pair stages of the precision form for D4S, whose polarisabilities depend on
// the partner's element: C6_ij = sum_w A_i[slot j][w] A_j[slot i][w], slots the
// distinct elements of the structure.
//
// A warp per atom i.  Its partners are taken in a list that groups them by slot,
// each slot's run padded to whole groups of eight lanes: every lane has a
// pair, whatever the elements (a loop over slots left most lanes idle and
// cost a trip per element), and the adjoint sums of a slot form over the eight lanes of
// a group by halving exchanges (21 for 24 frequencies).  The CTA makes the
// list of up to SL_TILE atoms in shared memory; slot data of atom i and the sums
// per slot (four copies, one per group of the warp) are there too.
//
// Bound by the latency of the gathered A_j and issue.  Measured, 96 structures of
// 20..147 atoms of 12 elements, against a loop over slots: C6 and two-body
// term 301 -> 99 us, ATM adjoints 189 -> 56 us.
#include "d4_common.cuh"
#include "d4_kernels.cuh"

namespace d4 {

namespace {

constexpr int SL_TILE = 1024;  // atoms per list
constexpr int SL_W = 24;       // frequencies, padded (eight lanes x 3)
constexpr int SL_WA = 28;      // row stride of atom i's slot data (no bank conflicts)
constexpr unsigned SL_NONE = 0xffffu;

// Halving exchanges over the lane bits 4, 2, 1: v[0 .. 2] end as the group's
// sums of values sl_first(lane) + 0 .. 2.
__device__ __forceinline__ void group_sums(float (&v)[SL_W]) {
  const int lane = threadIdx.x & 31;
#pragma unroll
  for (int s = 0; s < 3; ++s) {
    const int m = SL_W >> (s + 1), h = 4 >> s;
    const bool up = (lane & h) != 0;
#pragma unroll
    for (int q = 0; q < m; ++q) {
      const float keep = up ? v[q + m] : v[q];
      const float send = up ? v[q] : v[q + m];
      v[q] = keep + __shfl_xor_sync(0xffffffffu, send, h);
    }
  }
}
__device__ __forceinline__ int sl_first(int lane) {
  return 12 * ((lane >> 2) & 1) + 6 * ((lane >> 1) & 1) + 3 * (lane & 1);
}

// Slots that a structure can have, for everything in shared memory: a caller's S may
// be larger.
__host__ __device__ inline int sl_slots(const Ctx &c) {
  return c.S < MAX_ELEM_ID ? c.S : MAX_ELEM_ID;
}

__host__ __device__ inline int sl_entries(int S) { return SL_TILE + 8 * S; }
// shared memory: the list, slots of its groups and of the tile's atoms, run
// starts (in whole float4), then ``warp_floats`` per warp
__host__ __device__ inline size_t sl_list_bytes(int S) {
  const size_t b = 2 * (size_t)sl_entries(S) + sl_entries(S) / 8 + SL_TILE + 4 * (size_t)(S + 1);
  return (b + 31) & ~(size_t)15;
}

struct SlotList {
  unsigned short *at;    // atom of each entry relative to the tile, or SL_NONE
  unsigned char *group;  // slot of each group of eight entries
  unsigned char *slot;   // slot of each atom of the tile
  int *start;            // first entry of each slot's run
};

__device__ __forceinline__ SlotList slot_list_smem(void *p, int S) {
  SlotList l;
  l.start = reinterpret_cast<int *>(p);
  l.at = reinterpret_cast<unsigned short *>(l.start + S + 1);
  l.group = reinterpret_cast<unsigned char *>(l.at + sl_entries(S));
  l.slot = l.group + sl_entries(S) / 8;
  return l;
}

// The list of atoms t0 .. t0 + tn - 1 of structure b (all threads); returns
// its length.  Atoms keep their order within a slot.
__device__ int make_slot_list(const Ctx &c, int b, int t0, int tn, int nslot, const SlotList &l) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, W = blockDim.x >> 5;
  const size_t ab = (size_t)b * c.N + t0;
  __syncthreads();  // the last list is no longer read
  for (int k = threadIdx.x; k < tn; k += blockDim.x)
    l.slot[k] = c.w.z[ab + k] != 0 ? (unsigned char)c.w.slot[ab + k] : (unsigned char)255;
  __syncthreads();
  for (int s = warp; s < nslot; s += W) {
    int cnt = 0;
    for (int k = lane; k < ((tn + 31) & ~31); k += 32)
      cnt += __popc(__ballot_sync(0xffffffffu, k < tn && l.slot[k] == s));
    if (lane == 0) l.start[s + 1] = (cnt + 7) & ~7;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    l.start[0] = 0;
    for (int s = 0; s < nslot; ++s) l.start[s + 1] += l.start[s];
  }
  __syncthreads();
  for (int s = warp; s < nslot; s += W) {
    int o = l.start[s];
    const int end = l.start[s + 1];
    for (int g = o / 8 + lane; g < end / 8; g += 32) l.group[g] = (unsigned char)s;
    for (int k = lane; k < ((tn + 31) & ~31); k += 32) {
      const bool in = k < tn && l.slot[k] == s;
      const unsigned m = __ballot_sync(0xffffffffu, in);
      if (in) l.at[o + __popc(m & ((1u << lane) - 1u))] = (unsigned short)k;
      o += __popc(m);
    }
    if (o + lane < end) l.at[o + lane] = SL_NONE;
  }
  __syncthreads();
  return l.start[nslot];
}

// transposed index of (structure b, atom i, slot s, frequency w)
__device__ __forceinline__ size_t a32_at(const Ctx &c, int b, int i, int s, int w) {
  return (((size_t)b * c.S + s) * NFREQ + w) * c.N + i;
}

}  // namespace

namespace {

__host__ __device__ inline size_t fwd_floats(int S) {  // per warp
  return (size_t)S * (2 * SL_WA + 4 * SL_W);
}
__host__ __device__ inline size_t bwd_floats(int S) { return (size_t)S * 4 * SL_W; }

}  // namespace

// Fused C6 + BJ two-body term in FP32, the per-pair ATM table (float4:
// r^2, 1/r^2, (R0/r)^(alp/3), sqrt(C6(q=0)) / r^3), the direct gradient and
// the C6 adjoint.
template <bool GRAD, bool PGRAD>
__global__ void __launch_bounds__(256, 2) pair_fwd_d4s32_kernel(Ctx c) {
  const int b = blockIdx.y;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int i = blockIdx.x * (blockDim.x >> 5) + warp;
  const int N = c.N, n = c.w.n_eff[b], nslot = c.w.n_slots[b];
  extern __shared__ float4 s_dyn[];
  const int SS = sl_slots(c);
  const SlotList list = slot_list_smem(s_dyn, SS);
  // atom i's A at q and at q = 0 by slot, the adjoint sums by group and slot
  float *wa = reinterpret_cast<float *>(reinterpret_cast<char *>(s_dyn) + sl_list_bytes(SS)) +
              (size_t)warp * fwd_floats(SS);
  float *wa0 = wa + SS * SL_WA, *sums = wa0 + SS * SL_WA;
  const size_t ai = (size_t)b * N + (i < N ? i : 0);
  const int zi = i < n ? c.w.z[ai] : 0;
  const bool live = zi != 0;
  if (!live && i < N) {
    if (lane == 0) {
      c.out.d_energy[ai] = 0.0;
      if (GRAD) {
        c.out.d_gradient[3 * ai] = 0.0;
        c.out.d_gradient[3 * ai + 1] = 0.0;
        c.out.d_gradient[3 * ai + 2] = 0.0;
      }
    }
    if (GRAD && lane < NFREQ)
      for (int s = 0; s < c.S; ++s) c.w.G32[(ai * c.S + s) * NFREQ + lane] = 0.f;
  }
  const d4_params_t &p = c.par;
  const float s6 = c.pf.s6, s8 = c.pf.s8, s10 = c.pf.s10;
  const float cut2 = c.pf.cut2;
  const float4 *P = c.w.pos32 + (size_t)b * N;
  const float4 *PL = c.w.pos32lo + (size_t)b * N;
  const float4 pi = P[live ? i : 0], li = PL[live ? i : 0];
  const float wi = c.w.w32[ai];
  const int slot_i = c.w.slot[ai];
  float4 *T = c.w.ptf + (size_t)ai * N;
  float4 *Tda = PGRAD ? c.w.ptf_da + (size_t)ai * N : nullptr;
  // R0 = a1 sqrt(qq) + a2, qq = 3 r4r2_i r4r2_j, R0^6 and R0^8 as
  // double-floats, so that no FP32 rounding of a per-element-pair constant
  // biases every pair of that element pair the same way: from the per-call
  // element-pair table, or (per-atom r4r2 given) per pair from u_i = a1
  // sqrt(3) s_i, v_i = sqrt(3) s_i (FP64 per atom) and s_j = pos32.w + pos32lo.w
  const bool tabled = c.r4r2_in == nullptr;
  // compensated sums of c6 t6 (with (s10/s6) c10 t10 folded in) and of
  // c8 t8; s6 and s8 are applied in FP64 at the end (one FP32 sum of both
  // orders, with s8/s6 as a double-float, measured 4x less accurate)
  const double sref = p.s6 != 0.0 ? p.s6 : 1.0;
  const dfl rho10 = df_from(p.has_s10 ? p.s10 / sref : 0.0);
  const float rho6 = p.s6 != 0.0 ? 1.f : 0.f;
  Acc32 e_acc, e8_acc, gx, gy, gz;
  float pg[5] = {0.f, 0.f, 0.f, 0.f, 0.f};
  float r2mx = 0.f;  // largest r^2 of this atom's pairs (the ATM's far-atom test)
  if (live) {
    for (int s = 0; s < nslot; ++s) {
      // A' already carries sqrt((3/pi) w): C6 = sum_w A'_i A'_j
      if (lane < SL_WA) {
        const bool in = lane < NFREQ;
        wa[s * SL_WA + lane] = in ? c.w.A32[a32_at(c, b, i, s, lane)] : 0.f;
        wa0[s * SL_WA + lane] = in ? c.w.A032[a32_at(c, b, i, s, lane)] : 0.f;
      }
    }
    if (GRAD)
      for (int k = lane; k < 4 * SS * SL_W; k += 32) sums[k] = 0.f;
  }
  const float *Ab = c.w.A32 + a32_at(c, b, 0, slot_i, 0);
  const float *A0b = c.w.A032 + a32_at(c, b, 0, slot_i, 0);
  for (int t0 = 0; t0 < n; t0 += SL_TILE) {
    const int entries = make_slot_list(c, b, t0, min(SL_TILE, n - t0), nslot, list);
    if (!live) continue;
    for (int e0 = 0; e0 < entries; e0 += 32) {
      const int e = e0 + lane;
      const unsigned at = e < entries ? list.at[e] : SL_NONE;
      const int j = t0 + (int)at;
      const int sg = e < entries ? list.group[e >> 3] : 0;
      float K = 0.f, Ajr[NFREQ];
#pragma unroll
      for (int w = 0; w < NFREQ; ++w) Ajr[w] = 0.f;
      if (at != SL_NONE && j != i) {
        const size_t aj = (size_t)b * N + j;
        const int zj = c.w.z[aj];
        const float4 pj = P[j];
        const float3 d = pos_diff(pi, li, pj, PL[j]);
        const float dx = d.x, dy = d.y, dz = d.z;
        const float r2 = dx * dx + dy * dy + dz * dz;
        const float ir = __frcp_rn(sqrtf(r2));  // correctly rounded: no bias in the ATM records
        const float r = r2 * ir;
        float c6 = 0.f, c60 = 0.f;
#pragma unroll
        for (int w = 0; w < NFREQ; ++w) Ajr[w] = Ab[(size_t)w * N + j];
#pragma unroll
        for (int w = 0; w < NFREQ; ++w) {
          c6 = fmaf(wa[sg * SL_WA + w], Ajr[w], c6);
          c60 = fmaf(wa0[sg * SL_WA + w], A0b[(size_t)w * N + j], c60);
        }
        dfl R0d, qqd, R06d, R08d;
        if (tabled) {  // per element pair, from the table r4r2 values
          const float4 A = c.w.pairA[zi * MAX_ELEM_ID + zj], Bq = c.w.pairB[zi * MAX_ELEM_ID + zj];
          R0d = {A.x, A.y};
          qqd = {A.z, A.w};
          R06d = {Bq.x, Bq.y};
          R08d = {Bq.z, Bq.w};
        } else {  // per-atom r4r2 given (rare): FP64 per pair
          const double si = (double)pi.w + (double)li.w, sj = (double)pj.w + (double)PL[j].w;
          const double qq = 3.0 * si * si * sj * sj;
          const double R0 = p.a1 * sqrt(qq) + p.a2;
          const double R02 = R0 * R0, R06 = R02 * R02 * R02;
          R0d = df_from(R0);
          qqd = df_from(qq);
          R06d = df_from(R06);
          R08d = df_from(R06 * R02);
        }
        const float R0 = R0d.hi, sqq = sqrtf(qqd.hi);
        const float lnR0r = logf(R0 * ir) + R0d.lo / R0;
        const float ir2 = __frcp_rn(r2);
        T[j] = make_float4(r2, ir2, expf(c.pf.alp3 * lnR0r), sqrtf(c60) * (ir * ir2));
        if (GRAD && i < j) c.w.prSP32[(size_t)ai * N + j] = make_float2(0.f, 0.f);  // ATM sums
        r2mx = fmaxf(r2mx, r2);
        if (PGRAD) Tda[j] = make_float4(sqq / R0, 1.0f / R0, lnR0r, 0.f);
        if (r <= cut2) {
          const float r6 = r2 * r2 * r2, R02 = R0 * R0, R06 = R06d.hi;
          const float t6 = 1.0f / ((r6 + R06) + R06d.lo);
          float eterm = rho6 * c6 * t6;
          float dEdr = 6.0f * s6 * c6 * (r6 * ir) * t6 * t6;
          K = -s6 * t6;
          float dE_dR0 = 6.0f * s6 * c6 * (R06 / R0) * t6 * t6;
          pg[0] -= wi * c6 * t6;
          if (p.has_s8) {
            const float r8 = r6 * r2, R08 = R08d.hi, qq = qqd.hi;
            const float t8 = 1.0f / ((r8 + R08) + R08d.lo);
            const float c8 = fmaf(c6, qqd.hi, c6 * qqd.lo);
            const float e8 = c8 * t8;
            e8_acc.add(e8);
            dEdr += 8.0f * s8 * c8 * (r8 * ir) * t8 * t8;
            K -= s8 * qq * t8;
            dE_dR0 += 8.0f * s8 * c8 * (R08 / R0) * t8 * t8;
            pg[1] -= wi * c8 * t8;
          }
          if (p.has_s10) {  // rare: FP32 powers
            const float qq = sqq * sqq;
            const float r10 = r6 * r2 * r2, R010 = R06 * R02 * R02;
            const float t10 = 1.0f / (r10 + R010);
            const float q2 = qq * qq * (49.0f / 40.0f);
            const float c10 = c6 * q2;
            const float e10 = c10 * t10;
            eterm = fmaf(rho10.hi, e10, fmaf(rho10.lo, e10, eterm));
            dEdr += 10.0f * s10 * c10 * (r10 * ir) * t10 * t10;
            K -= s10 * q2 * t10;
            dE_dR0 += 10.0f * s10 * c10 * (R010 / R0) * t10 * t10;
            pg[2] -= wi * c10 * t10;
          }
          e_acc.add(eterm);
          const float phi = 0.5f * (wi + c.w.w32[aj]);
          dEdr *= phi;
          K *= phi;
          pg[3] += wi * 0.5f * dE_dR0 * sqq;
          pg[4] += wi * 0.5f * dE_dR0;
          const float f = dEdr * ir;
          gx.add(f * dx);
          gy.add(f * dy);
          gz.add(f * dz);
        }
      }
      if (GRAD) {
        float v[SL_W];
#pragma unroll
        for (int w = 0; w < SL_W; ++w) v[w] = w < NFREQ ? K * Ajr[w < NFREQ ? w : 0] : 0.f;
        group_sums(v);
        if (e < entries) {
          float *o = sums + ((lane >> 3) * SS + sg) * SL_W + sl_first(lane);
          o[0] += v[0];
          o[1] += v[1];
          o[2] += v[2];
        }
      }
    }
  }
  if (!live) return;
  if (GRAD) {  // dE/dA'_i
    __syncwarp();
    if (lane < NFREQ)
      for (int s = 0; s < c.S; ++s) {
        float g = 0.f;
        if (s < nslot)
          for (int k = 0; k < 4; ++k) g += sums[(k * SS + s) * SL_W + lane];
        c.w.G32[(ai * c.S + s) * NFREQ + lane] = g;
      }
  }
  const Acc32 ea = warp_sum_acc(e_acc), ea8 = warp_sum_acc(e8_acc);
  r2mx = warp_maxf(r2mx);
  if (lane == 0 && r2mx > 0.f) atomicMax(&c.w.atm_rowmax[ai], __float_as_uint(r2mx));
  if (PGRAD) {
    float v[5];
#pragma unroll
    for (int k = 0; k < 5; ++k) v[k] = warp_sumf(pg[k]);
    if (lane == 0) {
      atomicAdd(&c.w.pgrad[b * D4_PARAM_GRAD_STRIDE + 0], 0.5 * (double)v[0]);
      atomicAdd(&c.w.pgrad[b * D4_PARAM_GRAD_STRIDE + 1], 0.5 * (double)v[1]);
      atomicAdd(&c.w.pgrad[b * D4_PARAM_GRAD_STRIDE + 2], 0.5 * (double)v[2]);
      atomicAdd(&c.w.pgrad[b * D4_PARAM_GRAD_STRIDE + 3], (double)v[3]);
      atomicAdd(&c.w.pgrad[b * D4_PARAM_GRAD_STRIDE + 4], (double)v[4]);
    }
  }
  if (GRAD) {
    const Acc32 g0 = warp_sum_acc(gx), g1 = warp_sum_acc(gy), g2 = warp_sum_acc(gz);
    if (lane == 0) {
      c.out.d_gradient[3 * ai] = g0.value();
      c.out.d_gradient[3 * ai + 1] = g1.value();
      c.out.d_gradient[3 * ai + 2] = g2.value();
    }
  }
  if (lane == 0)
    c.out.d_energy[ai] = -0.5 * (sref * ea.value() + (p.has_s8 ? p.s8 * ea8.value() : 0.0));
}

// ATM forces, C6(q=0) adjoint, chain rule to dE/dCN and dE/dq, E2 + E3.
__global__ void __launch_bounds__(256) pair_bwd_d4s32_kernel(Ctx c) {
  const int b = blockIdx.y;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int x = blockIdx.x * (blockDim.x >> 5) + warp;
  const int N = c.N, n = c.w.n_eff[b], nslot = c.w.n_slots[b];
  extern __shared__ float4 s_dyn[];
  const int SS = sl_slots(c);
  const SlotList list = slot_list_smem(s_dyn, SS);
  float *sums = reinterpret_cast<float *>(reinterpret_cast<char *>(s_dyn) + sl_list_bytes(SS)) +
                (size_t)warp * bwd_floats(SS);  // by group and slot
  const size_t ax = (size_t)b * N + (x < N ? x : 0);
  const bool live = x < n && c.w.z[ax] != 0;
  if (!live && x < N && lane == 0) {
    c.w.dEdcn[ax] = 0.0;
    c.w.dEdq[ax] = 0.0;
    c.w.adj32[ax] = make_float4(0.f, 0.f, 0.f, 0.f);
  }
  const float4 *P = c.w.pos32 + (size_t)b * N;
  const float4 *PL = c.w.pos32lo + (size_t)b * N;
  const float4 px = P[live ? x : 0], lx = PL[live ? x : 0];
  const int slot_x = c.w.slot[ax];
  const size_t base = (size_t)b * N * N;
  const float4 *T = c.w.ptf + base + (size_t)(live ? x : 0) * N;
  const float *A0b = c.w.A032 + a32_at(c, b, 0, slot_x, 0);
  Acc32 gx, gy, gz;
  Acc32 dcn_acc, dq_acc;
  if (live)
    for (int k = lane; k < 4 * SS * SL_W; k += 32) sums[k] = 0.f;
  for (int t0 = 0; t0 < n; t0 += SL_TILE) {
    const int entries = make_slot_list(c, b, t0, min(SL_TILE, n - t0), nslot, list);
    if (!live) continue;
    for (int e0 = 0; e0 < entries; e0 += 32) {
      const int e = e0 + lane;
      const unsigned at = e < entries ? list.at[e] : SL_NONE;
      const int y = t0 + (int)at;
      const int sg = e < entries ? list.group[e >> 3] : 0;
      float v[SL_W];
#pragma unroll
      for (int w = 0; w < SL_W; ++w) v[w] = 0.f;
      if (at != SL_NONE && y != x) {
        const float2 sp = c.w.prSP32[base + (size_t)x * N + y];
        const float S = sp.x, Pv = sp.y;
        const float3 d = pos_diff(px, lx, P[y], PL[y]);
        gx.add(2.0f * S * d.x);
        gy.add(2.0f * S * d.y);
        gz.add(2.0f * S * d.z);
        if (Pv != 0.f) {
          const float cw = T[y].w;  // sqrt(C6(q=0)) / r^3: C6(q=0) = w^2 r^6
          const float r2 = d.x * d.x + d.y * d.y + d.z * d.z;
          const float D = Pv / (2.0f * (cw * cw) * (r2 * r2 * r2));
#pragma unroll
          for (int w = 0; w < NFREQ; ++w) v[w] = D * A0b[(size_t)w * N + y];
        }
      }
      group_sums(v);
      if (e < entries) {
        float *o = sums + ((lane >> 3) * SS + sg) * SL_W + sl_first(lane);
        o[0] += v[0];
        o[1] += v[1];
        o[2] += v[2];
      }
    }
  }
  if (!live) return;
  __syncwarp();
  // chain rule to CN and q (lane = frequency)
  if (lane < NFREQ)
    for (int s = 0; s < nslot; ++s) {
      const size_t o = (ax * c.S + s) * NFREQ + lane;
      float g0w = 0.f;  // dE/dA'0_x
      for (int k = 0; k < 4; ++k) g0w += sums[(k * SS + s) * SL_W + lane];
      const float gw = c.w.G32[o];
      const float *d = c.w.dA32 + 3 * o;
      dcn_acc.add(gw * d[0]);
      dcn_acc.add(g0w * d[2]);
      dq_acc.add(gw * d[1]);
    }
  const Acc32 g0 = warp_sum_acc(gx), g1 = warp_sum_acc(gy), g2 = warp_sum_acc(gz);
  const Acc32 dcn = warp_sum_acc(dcn_acc), dq = warp_sum_acc(dq_acc);
  if (lane == 0) {
    c.w.dEdcn[ax] = dcn.value();
    c.w.dEdq[ax] = dq.value();
    c.w.adj32[ax] = make_float4(dcn.hi + dcn.lo, 0.f, (float)c.w.q[ax], 0.f);
    c.out.d_gradient[3 * ax] += g0.value();
    c.out.d_gradient[3 * ax + 1] += g1.value();
    c.out.d_gradient[3 * ax + 2] += g2.value();
    c.out.d_energy[ax] += c.w.e3[ax];
  }
}

namespace {

// Eight warps per CTA share a list; fewer where many slots would not fit.
template <typename K>
void launch_slots(const Ctx &c, cudaStream_t st, K kernel, size_t warp_floats) {
  const size_t fixed = sl_list_bytes(sl_slots(c)), most = 200 * 1024;
  int warps = 8;
  while (warps > 1 && fixed + 4 * warps * warp_floats > most) --warps;
  const size_t smem = fixed + 4 * warps * warp_floats;
  if (smem > 48 * 1024) ensure_smem_impl(reinterpret_cast<const void *>(kernel), most);
  kernel<<<dim3((c.N + warps - 1) / warps, c.B), 32 * warps, smem, st>>>(c);
}

}  // namespace

void launch_pair_fwd_d4s32(const Ctx &c, cudaStream_t st) {
  const size_t f = fwd_floats(sl_slots(c));
  if (c.flags & D4_FLAG_PARAM_GRAD)
    launch_slots(c, st, pair_fwd_d4s32_kernel<true, true>, f);
  else if (c.flags & D4_FLAG_GRADIENT)
    launch_slots(c, st, pair_fwd_d4s32_kernel<true, false>, f);
  else
    launch_slots(c, st, pair_fwd_d4s32_kernel<false, false>, f);
}

void launch_pair_bwd_d4s32(const Ctx &c, cudaStream_t st) {
  launch_slots(c, st, pair_bwd_d4s32_kernel, bwd_floats(sl_slots(c)));
}

}  // namespace d4
