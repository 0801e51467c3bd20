// Q8_0 x Q8_0 weight matmul on the INT8 tensor cores: runq.c:317-342 evaluated exactly as written.
//
//   out[n, m] = sum_g  (float)( sum_{k in g} Wq[m,k] * Xq[n,k] )  *  Ws[m,g]  *  Xs[n,g]        (groups ascending)
//
// The inner integer sum of a group is ONE accumulator pass of tcgen05.mma.kind::i8 (int8 x int8 -> int32, exact;
// K = 32 per instruction, gs/32 instructions per group) with BOTH operands read straight from the TMA-written
// shared-memory tiles: no conversion warps, weights cross HBM and shared memory as the int8 bytes of the file.
// Each finished group accumulator [128 rows x NT columns] is pulled out of TMEM by the epilogue warps
// (thread = weight row), converted exactly, scaled by the row's weight scale and the column's activation scale in
// the reference's order and added in fp32 -- so without split-K the result is bit-identical to runq.c's loop
// (compiled without FMA contraction).
//   warp 0  TMA producer (weights first: they do not depend on the previous kernel)   warp 1  MMA issuer   warp 2  TMEM allocation
//   warps 4 on  epilogue: EW / 4 warps per 32-lane TMEM quarter, thread = weight row x its warp's share of the columns
// Rings: shared-memory SLOTS of [W 128x128 | X NTx128] int8 values (128 of K), TMEM STAGES of one slot's group sums, and the
// activation scales of a slot (a bulk copy of NT floats per group).
//
// What bounds it.  Few columns: the weights' way from HBM, 700 cycles per 16 KB slot and SM; every step of a slot's chain (producer, issuer, read-out)
// has to stay below that, so the issuer and the producer are one elected thread each that counts instead of dividing.  Many columns: the epilogue,
// 16384 sums per slot of 64 columns to convert, scale twice and add (1700 instructions a slot besides what the hand-over of a slot takes,
// which is paid per warp: hence few warps with many columns, and U columns of one group at a time with the next U already on their way out of TMEM).
// Two or three epilogue warps a scheduler leave a third of the issue slots empty.  At 4096 of K and 64 values a group, us, before (two issuers, 16 warps with
// all of a slot in registers, the item's scales staged between two barriers) and now: 930 rows x 12288 293 -> 171, 64 x 32000 66.5 -> 43.7,
// 32 x 32000 41.5 -> 33.5, 1 x 12288 19.6 -> 17.6; 930 x 4096 x 11008 290 -> 158.  64 columns by 16 warps instead of 8: 253 for the first of these.
// mma.sync instead, with the sums in registers: 329, and 29.8 for one row.
#include <cuda.h>

#include <type_traits>

#include "common.cuh"
#include "gemm_tc.h"
#include "ktrace.cuh"
#include "tc_common.cuh"
#include "workspace.h"

namespace tha {

struct Q8iP {
  int M[3]; int tiles[3]; int out_off[3];
  const float* S[3];                 // weight group scales [M, ngrp]
  const float* xsT; int ldxs;        // activation group scales, transposed: xsT[g * ldxs + n]
  int K, N, ny, gs, ngrp;
  int slots_total, slots_per_split;  // ring slots of 128 values
  float* out; long long ldo; long long zstride;
  int* error_flag;
  int nring, nacc, nxs;              // slots, TMEM stages (a power of two) and scale buffers in use
  int splits, n_items;               // work items = (tiles of all matrices) x column tiles x splits
};

template <int NT>
struct Q8iSmem {
  static constexpr int W_BYTES = TC_BM * 128, X_BYTES = NT * 128, SLOT = W_BYTES + X_BYTES;
  static constexpr int TMEM_COLS = 512;
  static constexpr int NRING_MAX = 10, NACC_MAX = 32;
  static constexpr int NXS_MAX = 64;              // a power of two >= NRING_MAX + NACC_MAX + 1
  static constexpr int NMD = 64;                  // commit barriers (more than the slots that can be in flight)
  static constexpr int BARS = (NRING_MAX + NMD + NACC_MAX + NXS_MAX) * 8 + 64;
  static_assert(NRING_MAX + NACC_MAX + 1 <= NMD, "commit barrier ring too short");
};

__host__ __device__ constexpr uint32_t q8i_idesc(int nt) {   // kind::i8: D = S32 (2), A = B = signed 8-bit (1), K-major, M = 128
  return (2u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(nt >> 3) << 17) | ((uint32_t)(TC_BM >> 4) << 24);
}
__device__ __forceinline__ void q8i_mma(uint32_t tmem_d, uint64_t adesc, uint64_t bdesc, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::i8 [%0], %1, %2, %3, p;\n\t}"
      ::"r"(tmem_d), "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate) : "memory");
}
__device__ __forceinline__ void q8i_bulk(void* dst, const void* src, unsigned bytes, uint64_t* bar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
               ::"r"(tc_smem_u32(dst)), "l"(src), "r"(bytes), "r"(tc_smem_u32(bar)) : "memory");
}
__device__ __forceinline__ void q8i_wait_ld() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }
__device__ __forceinline__ void q8i_ld(uint32_t taddr, uint32_t (&v)[16]) { tc_tmem_ld16(taddr, v); }
__device__ __forceinline__ void q8i_ld(uint32_t taddr, uint32_t (&v)[8]) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
               : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]) : "r"(taddr));
}
__device__ __forceinline__ unsigned long long q8i_pair(float a, float b) {
  unsigned long long r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
  return r;
}
__device__ __forceinline__ unsigned long long q8i_mul2(unsigned long long a, unsigned long long b) {
  unsigned long long r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
// the sums stay scalar: a packed add behind a packed multiply is contracted
__device__ __forceinline__ void q8i_add(float& a0, float& a1, unsigned long long p) {
  float p0, p1;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(p0), "=f"(p1) : "l"(p));
  a0 = __fadd_rn(a0, p0);
  a1 = __fadd_rn(a1, p1);
}
__device__ __forceinline__ bool q8i_try(uint32_t bar, unsigned parity) {
  unsigned ok;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(ok) : "r"(bar), "r"(parity) : "memory");
  return ok != 0;
}
// All lanes wait for two barriers; the answer is the warp's.
__device__ __forceinline__ bool q8i_warp_wait2(uint32_t b0, unsigned ph0, uint32_t b1, unsigned ph1, int* abort_flag) {
  const bool o0 = q8i_try(b0, ph0), o1 = q8i_try(b1, ph1);
  if (__all_sync(THA_FULL_MASK, o0 && o1)) return true;
  for (unsigned n = 0; !__all_sync(THA_FULL_MASK, q8i_try(b0, ph0) && q8i_try(b1, ph1)); n++) {
    if (n > (1u << 22)) *((volatile int*)abort_flag) = 1;
    if ((n & 1023u) == 1023u && __any_sync(THA_FULL_MASK, *((volatile int*)abort_flag) != 0)) return false;
  }
  return true;
}
__device__ __forceinline__ void q8i_lds4(uint32_t addr, unsigned long long& x, unsigned long long& y) {
  asm volatile("ld.shared.v2.u64 {%0, %1}, [%2];" : "=l"(x), "=l"(y) : "r"(addr));
}

// Persistent: a CTA walks the work items (weight tile, column tile, K split) blockIdx.x, blockIdx.x + gridDim.x, ...
// with ONE running slot counter, so the TMA ring, the MMA issuer and the epilogue flow from one item into the next
// without draining (a fresh CTA per item paid ~3 us of ramp for ~6 us of streaming).
template <int NT, int EW, int GPS>
__global__ void __launch_bounds__(128 + 32 * EW, 1)
gemm_q8i_kernel(const __grid_constant__ CUtensorMap mw0, const __grid_constant__ CUtensorMap mw1,
                const __grid_constant__ CUtensorMap mw2, const __grid_constant__ CUtensorMap mx, const Q8iP p) {
  using S = Q8iSmem<NT>;
  extern __shared__ unsigned char tc_smem_raw[];
  unsigned char* smem = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(tc_smem_raw) + 1023) & ~(uintptr_t)1023);
  const int nring = p.nring, nacc = p.nacc, nxs = p.nxs;
  constexpr int gps_sh = GPS == 4 ? 2 : GPS - 1;
  float* xs_sm = reinterpret_cast<float*>(smem + nring * S::SLOT);   // [nxs][GPS][NT]
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + nring * S::SLOT + nxs * GPS * NT * 4);
  uint64_t* full = bars;                       // slot landed (W + X bytes)
  uint64_t* mdone = full + S::NRING_MAX;       // the MMAs of a slot have completed: slot reusable, group sums readable
  uint64_t* aempty = mdone + S::NMD;           // a stage's group sums have been read out by all epilogue warps
  uint64_t* xfull = aempty + S::NACC_MAX;      // a slot's activation scales have landed
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(xfull + S::NXS_MAX);
  int* abort_flag = reinterpret_cast<int*>(tmem_slot + 1);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int tiles01 = p.tiles[0] + p.tiles[1];
  __shared__ int kt_q8_s;

  // work item -> (matrix, row0, n0, first slot, slots, groups)
  struct Item { int mat, row0, n0, slot0, nslots, ng; };
  auto item_of = [&](int it) -> Item {
    Item w;
    const int z = it % p.splits;
    const int t = it / p.splits;
    int tile = t / p.ny;
    w.n0 = (t - tile * p.ny) * NT;
    w.mat = 0;
    if (tile >= p.tiles[0]) { w.mat = 1; if (tile >= tiles01) { w.mat = 2; tile -= tiles01; } else tile -= p.tiles[0]; }
    w.row0 = tile * TC_BM;
    w.slot0 = z * p.slots_per_split;
    w.nslots = p.slots_total - w.slot0;
    if (w.nslots > p.slots_per_split) w.nslots = p.slots_per_split;
    w.ng = p.ngrp - (w.slot0 << gps_sh);
    if (w.ng > (w.nslots << gps_sh)) w.ng = w.nslots << gps_sh;
    return w;
  };

  if (threadIdx.x == 0) {
    for (int s = 0; s < nring; s++) tc_mbar_init(&full[s], 1);
    for (int b = 0; b < S::NMD; b++) tc_mbar_init(&mdone[b], 1);
    for (int b = 0; b < nacc; b++) tc_mbar_init(&aempty[b], EW);
    for (int b = 0; b < nxs; b++) tc_mbar_init(&xfull[b], 1);
    *abort_flag = 0;
    kt_q8_s = kt_begin((unsigned long long)KT_GEMM_Q8 | ((unsigned long long)p.splits << 16) | ((unsigned long long)p.n_items << 32));
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  }
  if (warp == 0 && lane == 0) {
    asm volatile("prefetch.tensormap [%0];" ::"l"(&mw0) : "memory");
    if (p.tiles[1]) asm volatile("prefetch.tensormap [%0];" ::"l"(&mw1) : "memory");
    if (p.tiles[2]) asm volatile("prefetch.tensormap [%0];" ::"l"(&mw2) : "memory");
    asm volatile("prefetch.tensormap [%0];" ::"l"(&mx) : "memory");
  }
  if (warp == 2) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(tc_smem_u32(tmem_slot)), "r"(S::TMEM_COLS));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::);
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem_base = *tmem_slot;
  const int kt = kt_q8_s;

  if (warp == 0) {
    // ===== TMA producer
    if (tc_elect()) {
      uint64_t pol_w;
      asm volatile("createpolicy.fractional.L2::evict_first.b64 %0, 1.0;" : "=l"(pol_w));
      int jb = 0;                                   // running slot counter at the start of the item
      int xr = 0, s = 0;                            // running scale buffer and ring slot
      int sent = 0;
      bool ok = true;
      for (int it = blockIdx.x; it < p.n_items && ok; it += gridDim.x) {
        const Item w = item_of(it);
        const CUtensorMap* mw = (w.mat == 0) ? &mw0 : (w.mat == 1 ? &mw1 : &mw2);
        const int left = p.ldxs - w.n0;
        const unsigned xbytes = 4u * (unsigned)(left < NT ? left : NT);   // rows of scales are padded to ldxs, not always to the tile
        auto activations = [&](int j) {      // the X tile of slot j and its groups' scales
          tc_mbar_expect_tx(&full[s], S::SLOT);
          tc_tma_2d(smem + s * S::SLOT + S::W_BYTES, &mx, (w.slot0 + j) * 32, w.n0, &full[s]);
          int n = w.ng - (j << gps_sh);
          if (n > GPS) n = GPS;
          tc_mbar_expect_tx(&xfull[xr], n * xbytes);
          const float* src = p.xsT + (size_t)((w.slot0 + j) << gps_sh) * p.ldxs + w.n0;
          for (int g = 0; g < n; g++) q8i_bulk(xs_sm + ((xr << gps_sh) + g) * NT, src + (size_t)g * p.ldxs, xbytes, &xfull[xr]);
          if (++xr == nxs) xr = 0;
          if (++s == nring) s = 0;
        };
        int j = 0;
        if (jb == 0) {
          // the first ring of weight tiles goes out before the dependency wait (transaction bytes may land before
          // the matching expect_tx: the phase cannot complete until the arrival below)
          const int pre = w.nslots < nring ? w.nslots : nring;
          for (; j < pre; j++) tc_tma_2d_hint(smem + j * S::SLOT, mw, (w.slot0 + j) * 32, w.row0, &full[j], pol_w);
          pdl_wait();
          kt_stamp(kt, 1);
          for (j = 0; j < pre; j++) activations(j);
        }
        for (; j < w.nslots; j++) {
          const int jg = jb + j;
          if (jg >= nring) {
            // The slot use whose MMAs must have completed.  They began when the stage nacc uses earlier had been read out, and a warp has
            // read a stage out only behind its last use of the scales before it: with nring + nacc + 1 scale buffers the next is free too.
            const int st = jg - nring;
            if (!tc_mbar_wait(&mdone[st % S::NMD], (st / S::NMD) & 1u, abort_flag)) { ok = false; sent = jg; break; }
          }
          tc_tma_2d_hint(smem + s * S::SLOT, mw, (w.slot0 + j) * 32, w.row0, &full[s], pol_w);
          activations(j);
        }
        jb += w.nslots;
      }
      if (!ok) {
        tc_drain(full, nring, sent);
        tc_drain(xfull, nxs, sent);
      }
    }
    __syncwarp();
  } else if (warp == 1) {
    // ===== MMA issuer: one thread, with counters instead of divisions -- its turn (wait, wait, four MMAs, commit) is what a slot takes at least
    if (tc_elect()) {
      constexpr uint32_t idesc = q8i_idesc(NT);
      constexpr int MPG = 4 / GPS;               // MMAs per group
      const uint64_t adesc0 = tc_smem_desc(tc_smem_u32(smem));
      int jg = 0, s = 0, stage = 0;
      unsigned fph = 0, aph = 1;
      bool ok = true;
      for (int it = blockIdx.x; it < p.n_items && ok; it += gridDim.x) {
        const int nslots = item_of(it).nslots;
        for (int j = 0; j < nslots; j++) {
          // a stage is empty the first time around: the wait for the phase before the first passes
          if (!tc_mbar_wait(&aempty[stage], aph, abort_flag) || !tc_mbar_wait(&full[s], fph, abort_flag)) { ok = false; break; }
          if (jg == 0) kt_stamp(kt, 2);
          asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
          const uint64_t adesc = adesc0 + (uint64_t)(s * (S::SLOT >> 4)), bdesc = adesc + (uint64_t)(S::W_BYTES >> 4);
          const uint32_t acc0 = tmem_base + (uint32_t)(stage * GPS * NT);
#pragma unroll
          for (int sub = 0; sub < 4; sub++)       // past the end of K the tiles are zero-filled: always four MMAs
            q8i_mma(acc0 + (uint32_t)(sub / MPG * NT), adesc + (uint64_t)(sub * 2), bdesc + (uint64_t)(sub * 2), idesc,
                    (uint32_t)(sub % MPG != 0));
          tc_commit(&mdone[jg & (S::NMD - 1)]);
          jg++;
          if (++s == nring) { s = 0; fph ^= 1u; }
          if (++stage == nacc) { stage = 0; aph ^= 1u; }
        }
      }
      kt_stamp(kt, 3);
    }
    __syncwarp();
  } else if (warp >= 4) {
    // ===== epilogue: thread = weight row (TMEM lane) x CH columns, U columns of one group at a time; the next U are on their way out of
    // TMEM while these are scaled and added
    constexpr int CH = NT * 4 / EW, U = CH < 16 ? CH : 16, NU = CH / U;
    const int q = warp & 3;
    const int c0 = ((warp - 4) >> 2) * CH;       // first column of this warp's share
    const int r = q * 32 + lane;
    const uint32_t tq = tmem_base + ((uint32_t)(q * 32) << 16) + (uint32_t)c0;
    const uint32_t xs0 = tc_smem_u32(xs_sm) + (uint32_t)c0 * 4, mdone0 = tc_smem_u32(mdone), xfull0 = tc_smem_u32(xfull), aempty0 = tc_smem_u32(aempty);
    const int nxs_sh = 31 - __clz(nxs);
    pdl_trigger();
    pdl_wait();                                     // the output may still be read by the previous kernel
    unsigned jg = 0;                                // running slot
    bool ok = true;
    uint32_t v[2][U];
    for (int it = blockIdx.x; it < p.n_items && ok; it += gridDim.x) {
      const Item w = item_of(it);
      const int ng = w.ng;
      const int row = w.row0 + r;
      const bool row_ok = row < p.M[w.mat];
      const float* srow = p.S[w.mat] + (size_t)(row_ok ? row : p.M[w.mat] - 1) * p.ngrp + (w.slot0 << gps_sh);
      float acc[CH];
#pragma unroll
      for (int c = 0; c < CH; c++) acc[c] = 0.0f;
      // Weight scales: this thread's row, four groups per 128-bit load, requested two to three chunks (8-12 groups) before their use --
      // with ~200 KB of the SM's memory carved out as shared, L1 keeps next to nothing and every one of these loads is an L2 round trip.
      const bool ws_vec = ((reinterpret_cast<uintptr_t>(srow) & 15u) == 0) && (p.ngrp % 4 == 0);
      auto load_ws4 = [&](int g) -> float4 {
        float4 r4 = make_float4(0.f, 0.f, 0.f, 0.f);
        if (g + 3 < ng && ws_vec) return __ldg(reinterpret_cast<const float4*>(srow + g));
        if (g < ng) r4.x = __ldg(srow + g);
        if (g + 1 < ng) r4.y = __ldg(srow + g + 1);
        if (g + 2 < ng) r4.z = __ldg(srow + g + 2);
        if (g + 3 < ng) r4.w = __ldg(srow + g + 3);
        return r4;
      };
      float4 ws_n1 = load_ws4(0), ws_n2 = load_ws4(4), ws_n3 = load_ws4(8);
      uint32_t ta, xs;
      auto slot_ready = [&]() {   // the running slot's sums and scales
        const unsigned x = jg & (unsigned)(nxs - 1);
        if (!q8i_warp_wait2(mdone0 + (jg & (S::NMD - 1)) * 8, (jg / S::NMD) & 1u, xfull0 + x * 8, (jg >> nxs_sh) & 1u, abort_flag)) ok = false;
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        ta = tq + (jg & (unsigned)(nacc - 1)) * (GPS * NT);
        xs = xs0 + x * (GPS * NT * 4);
      };
      // group k of a chunk: `end` = the item's last
      auto group = [&](auto kc, float ws, bool end) {
        constexpr int k = decltype(kc)::value;
        const unsigned long long ws2 = q8i_pair(ws, ws);
#pragma unroll
        for (int u = 0; u < NU; u++) {
          uint32_t (&cur)[U] = v[(k * NU + u) & 1];
          uint32_t (&nxt)[U] = v[(k * NU + u + 1) & 1];
          unsigned long long x[U / 2];
#pragma unroll
          for (int c = 0; c < U; c += 4) q8i_lds4(xs + (uint32_t)(k % GPS * NT + u * U + c) * 4, x[c / 2], x[c / 2 + 1]);   // one address a warp
          q8i_wait_ld();
          if (u < NU - 1) {
            q8i_ld(ta + (uint32_t)(k % GPS * NT + (u + 1) * U), nxt);
          } else if ((k + 1) % GPS == 0 || end) {   // the slot's sums have all been read
            asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
            __syncwarp();
            if (lane == 0)
              asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(aempty0 + (jg & (unsigned)(nacc - 1)) * 8) : "memory");
            jg++;
            if (!end) {
              slot_ready();
              q8i_ld(ta, nxt);
            }
          } else {
            q8i_ld(ta + (uint32_t)((k % GPS + 1) * NT), nxt);
          }
          // runq.c:334 in its order: (sum * weight scale) * activation scale, added; each rounded by itself
#pragma unroll
          for (int c = 0; c < U; c += 2) {
            const unsigned long long f = q8i_pair(__int2float_rn((int)cur[c]), __int2float_rn((int)cur[c + 1]));
            q8i_add(acc[u * U + c], acc[u * U + c + 1], q8i_mul2(q8i_mul2(f, ws2), x[c / 2]));
          }
        }
      };
      slot_ready();
      if (jg == 0 && threadIdx.x == 128) kt_stamp(kt, 4);
      q8i_ld(ta, v[0]);
      int gc = 0;
      for (; gc + 4 <= ng; gc += 4) {
        const float4 w4 = ws_n1;
        ws_n1 = ws_n2; ws_n2 = ws_n3;
        ws_n3 = load_ws4(gc + 12);
        group(std::integral_constant<int, 0>(), w4.x, false);
        group(std::integral_constant<int, 1>(), w4.y, false);
        group(std::integral_constant<int, 2>(), w4.z, false);
        group(std::integral_constant<int, 3>(), w4.w, gc + 4 == ng);
      }
      if (gc < ng) {
        group(std::integral_constant<int, 0>(), ws_n1.x, gc + 1 == ng);
        if (gc + 1 < ng) group(std::integral_constant<int, 1>(), ws_n1.y, gc + 2 == ng);
        if (gc + 2 < ng) group(std::integral_constant<int, 2>(), ws_n1.z, true);
      }
      float* outz = p.out + (size_t)(it % p.splits) * p.zstride + p.out_off[w.mat] + row;
      if (ok && row_ok) {
#pragma unroll
        for (int c = 0; c < CH; c++) {
          const int n = w.n0 + c0 + c;
          if (n < p.N) outz[(size_t)n * p.ldo] = acc[c];
        }
      }
      if (it == (int)blockIdx.x && threadIdx.x == 128) kt_stamp(kt, 5);
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  }
  __syncthreads();
  if (threadIdx.x == 0) kt_stamp(kt, 6);
  if (warp == 2) {
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(S::TMEM_COLS));
  }
  if (threadIdx.x == 0 && *abort_flag && p.error_flag) *((volatile int*)p.error_flag) = 1;
}

bool gemm_q8i_ok(const Q8iArgs& a) {
  if (a.gs != 32 && a.gs != 64 && a.gs != 128) return false;
  if (a.K % a.gs || a.K < 128 || a.K % 16 || a.N < 1 || a.n_mats < 1 || a.n_mats > 3 || !a.Xq || !a.xsT || !a.out) return false;
  if ((reinterpret_cast<uintptr_t>(a.Xq) & 15u) || (reinterpret_cast<uintptr_t>(a.xsT) & 15u) || a.ldxs % 4) return false;
  for (int i = 0; i < a.n_mats; i++)
    if (!a.Wq[i] || !a.Ws[i] || (reinterpret_cast<uintptr_t>(a.Wq[i]) & 15u) || a.M[i] < 1) return false;
  return true;
}

// The column tile by which callers size their scale rows and plan their splits (a split is part of a result's bits: the plan stays).
int gemm_q8i_pick_nt(int N, int gs) {
  const int nt = N <= 16 ? 16 : (N <= 32 ? 32 : 64);
  return nt > gs ? gs : nt;
}

// The column tile that a launch takes: the narrowest that holds all columns; past 64 the one whose rounds over the SMs cost least.  A slot takes
// 1080 cycles with 64 columns, 1450 with 96, 1910 with 128 (measured at 930 rows x 12288 x 4096: 182, 171 and 193 us of 10, 7 and 6 rounds; x 4096 x 4096:
// 75, 76 and 70 us).  At 32 values a group two stages of 96 columns do not fit TMEM.
static int q8i_tile(int N, int gs, int tiles_splits, int sms) {
  if (N <= 64) return N <= 16 ? 16 : (N <= 32 ? 32 : 64);
  constexpr int width[3] = {64, 96, 128}, cost[3] = {1080, 1450, 1910};
  int best = 64;
  long long least = -1;
  for (int i = 0; i < (gs == 32 ? 1 : 3); i++) {
    const long long c = (long long)ceil_div(tiles_splits * ceil_div(N, width[i]), sms) * cost[i];
    if (least < 0 || c < least) { least = c; best = width[i]; }
  }
  return best;
}

template <int NT, int EW, int GPS>
static int q8i_launch_gs(cudaStream_t st, const CUtensorMap* mw, const CUtensorMap& mx, Q8iP& p, int sms, bool pdl) {
  using S = Q8iSmem<NT>;
  static_assert(2 * GPS * NT <= S::TMEM_COLS, "two stages of group sums at least");
  p.nacc = 2;
  while (2 * p.nacc * GPS * NT <= S::TMEM_COLS && 2 * p.nacc <= S::NACC_MAX) p.nacc *= 2;
  constexpr int XS_BYTES = GPS * NT * 4;
  for (p.nring = S::NRING_MAX;; p.nring--) {   // the longest ring that fits beside its scale buffers
    for (p.nxs = 1; p.nxs < p.nring + p.nacc + 1;) p.nxs *= 2;
    if (p.nring * S::SLOT + p.nxs * XS_BYTES + S::BARS + 1024 /*alignment*/ + 64 /*static*/ <= TC_SMEM_LIMIT) break;
  }
  const size_t smem = (size_t)p.nring * S::SLOT + (size_t)p.nxs * XS_BYTES + S::BARS + 1024;
  auto k = gemm_q8i_kernel<NT, EW, GPS>;
  THA_CUDA_OK(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  THA_CUDA_OK(launch(k, dim3(p.n_items < sms ? p.n_items : sms), dim3(128 + 32 * EW), smem, st, pdl, mw[0], mw[1], mw[2], mx, p));
  return THA_STATUS_SUCCESS;
}
template <int NT, int EW>
static int q8i_launch_nt(cudaStream_t st, const CUtensorMap* mw, const CUtensorMap& mx, Q8iP& p, int sms, bool pdl) {
  if (p.gs == 128) return q8i_launch_gs<NT, EW, 1>(st, mw, mx, p, sms, pdl);
  if (p.gs == 64) return q8i_launch_gs<NT, EW, 2>(st, mw, mx, p, sms, pdl);
  if constexpr (NT <= 64) return q8i_launch_gs<NT, EW, 4>(st, mw, mx, p, sms, pdl);
  return THA_STATUS_NOT_SUPPORTED;
}

int gemm_q8i_launch(cudaStream_t st, const Q8iArgs& a, bool pdl) {
  if (!gemm_q8i_ok(a)) return THA_STATUS_INVALID_ARG;
  const int plan_nt = gemm_q8i_pick_nt(a.N, a.gs);
  if (a.ldxs < ceil_div(a.N, plan_nt) * plan_nt) return THA_STATUS_INVALID_ARG;
  CUtensorMap mw[3], mx;
  Q8iP p = {};
  int tiles = 0;
  for (int i = 0; i < 3; i++) {
    if (i < a.n_mats) {
      THA_TRY_RC(tc_map(a.Wq[i], a.M[i], a.K, a.K, TC_BM, &mw[i], 1));
      p.M[i] = a.M[i]; p.tiles[i] = ceil_div(a.M[i], TC_BM); p.out_off[i] = a.out_off[i]; p.S[i] = a.Ws[i];
    } else {
      mw[i] = mw[0];
    }
    tiles += p.tiles[i];
  }
  p.xsT = a.xsT; p.ldxs = a.ldxs; p.K = a.K; p.N = a.N; p.gs = a.gs; p.ngrp = a.K / a.gs;
  p.slots_total = ceil_div(a.K, 128);
  const int splits = a.splits < 1 ? 1 : a.splits;
  p.slots_per_split = ceil_div(p.slots_total, splits);
  if (ceil_div(p.slots_total, p.slots_per_split) != splits) return THA_STATUS_INVALID_ARG;
  {  // The longest split that is served: an item's scales ([groups][planned tile] floats) beside three slots of the planned tile in 220 KB.  The scales
     // travel with their slots now and set no limit; what calls are refused is as it was.
    const int slot = TC_BM * 128 + plan_nt * 128, sb = a.gs / plan_nt;
    const int fit = (TC_SMEM_LIMIT - 3072) / slot > 10 ? 10 : (TC_SMEM_LIMIT - 3072) / slot;
    if (fit - ceil_div(ceil_div(p.slots_per_split, sb) * sb * (128 / a.gs) * plan_nt * 4, slot) < 3) return THA_STATUS_NOT_SUPPORTED;
  }
  p.out = a.out; p.ldo = a.ldo; p.zstride = a.zstride;
  THA_TRY_RC(gemm_tc_init(&p.error_flag));
  const int sms = sm_budget();
  const int NT = q8i_tile(a.N, a.gs, tiles * splits, sms);
  THA_TRY_RC(tc_map(a.Xq, a.N, a.K, a.K, NT, &mx, 1));
  p.ny = ceil_div(a.N, NT);
  p.splits = splits;
  p.n_items = tiles * p.ny * splits;
  switch (NT) {
    case 16: return q8i_launch_nt<16, 4>(st, mw, mx, p, sms, pdl);
    case 32: return q8i_launch_nt<32, 8>(st, mw, mx, p, sms, pdl);
    case 64: return q8i_launch_nt<64, 8>(st, mw, mx, p, sms, pdl);
    case 96: return q8i_launch_nt<96, 12>(st, mw, mx, p, sms, pdl);
    default: return q8i_launch_nt<128, 8>(st, mw, mx, p, sms, pdl);
  }
}

}  // namespace tha
