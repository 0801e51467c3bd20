// bf16 weight matmul on the tensor cores: tcgen05.mma.kind::f16 (bf16 x bf16 -> fp32 in TMEM) with BOTH operands read
// straight from TMA-written shared memory -- no conversion warps, the weights cross HBM and shared memory as the two
// bytes per value they are stored in.
//
//   out[n, row] = sum_k W[row, k] * X[n, k]      W: [M, K] row-major bf16, X: [N, K] row-major bf16 (rows = slots or
//                                                prompt positions, already rounded to bf16 by the producing kernel)
//
// This is the matmul of the bf16 model path (the reference declares the 16-bit
// weight structs at include/models.hpp:77-117 and never fills them) for more than 8 rows and for prompt ingestion, where
// the fp32 path's 3xTF32 scheme spends three tensor-core passes and a converter stage per useful one.
//
// Structure (persistent: 148 CTAs walk (weight tile, column tile, K split) items with running ring counters):
//   warp 0   TMA producer: per k-block of 64 values (one 128-byte swizzle row) the W tile [128 x 64] and the X tile
//            [NT x 64] into a ring of up to 8 stages; the first ring of W tiles goes out before griddepcontrol.wait
//   warp 1   MMA issuer: 4 x (M 128, N NT, K 16) per stage; tcgen05.commit frees the stage; the accumulator is DOUBLE
//            buffered in TMEM (2 x NT columns), so the next item's MMAs run while the epilogue drains the previous one
//   warp 2   TMEM allocation
//   warps 4-7  epilogue: thread = weight row (TMEM lane), 16 columns per tcgen05.ld, optional column scale, coalesced
//            stores (a warp writes 32 consecutive rows of one column); split-K partials to out + z * zstride
// Up to three matrices with the same K are stacked in one launch (wq|wk|wv, w1|w3); or up to BF_MAX_MATS row ranges of one matrix, each
// with activation rows of its own (BfArgs::stacked): an item's TMA coordinates start at its matrix's first weight and activation row,
// rows of a neighbouring range that a ragged tile brings along are not stored.
#include <stdlib.h>

#include "gemm_tc.h"
#include "hybrid_ops.cuh"
#include "tc_common.cuh"

namespace tha {

constexpr int BF_THREADS = 256;
constexpr int BF_BK = 64;             // bf16 values per k-block: 128 bytes

struct BfP {
  int M[BF_MAX_MATS]; int tiles[BF_MAX_MATS]; int out_off[BF_MAX_MATS]; int w_row[BF_MAX_MATS]; int x_row[BF_MAX_MATS];
  int n_mats, stacked;
  int K, N, ny, kblocks_total, kblocks_per_split;
  float* out; long long ldo; long long zstride;
  const float* colscale;
  int* error_flag;
  int splits, n_items;
  uint16_t* act_out; long long ld_act;         // kernels with an activation in the read-out
  int act; float act_limit, act_alpha;         // BF_GATED, BF_UNGATED: THA_ACT_*
};
// what a work item's read-out does with its accumulators
enum { BF_PLAIN = 0, BF_SWIGLU = 1, BF_GATED = 2, BF_UNGATED = 3 };

// MT = weight tiles of 128 rows per work item.  MT = 2 (prompt-sized N only): a CTA multiplies 256 weight rows by the
// same 256 activation columns -- per 64-value k-block it pulls 32 + 32 KB through L2 for twice the flops of the 16 + 32 KB
// of a 128-row tile.  With 128 x 256 tiles the prompt matmuls were bound by L2 -> shared-memory traffic (768 MB per
// 4096 x 4096 x 2048 matmul, ~48 % of the sustained tensor peak); the two accumulators then fill all 512 TMEM columns, so
// the read-out of an item is no longer hidden behind the next item's MMAs (eight warps keep it at a few per cent).
template <int NT, int MT = 1>
struct BfSmem {
  static constexpr int W_BYTES = MT * TC_BM * 128, X_BYTES = NT * 128, STAGE = W_BYTES + X_BYTES;
  static constexpr int NST_RAW = (TC_SMEM_LIMIT - 2048) / STAGE;
  static constexpr int NST = NST_RAW > 8 ? 8 : NST_RAW;
  static constexpr int NBUF = (2 * MT * NT <= 512) ? 2 : 1;           // accumulator buffers of MT x NT columns
  static constexpr int TMEM_COLS = NBUF * MT * NT < 32 ? 32 : NBUF * MT * NT;   // powers of two: NT in {16, 32, 64, 128, 256}
  static constexpr int TOTAL = NST * STAGE + 1024 + (2 * NST + 4) * 8 + 64;
  static_assert(NST >= 3, "ring too short");
  static_assert(TOTAL <= TC_SMEM_LIMIT, "shared memory overflow");
};

// kind::f16 with bf16 operands, fp32 accumulate, both K-major, M = 128, N = nt (cute::UMMA::InstrDescriptor)
__host__ __device__ constexpr uint32_t bf_idesc(int nt) {
  return (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(nt >> 3) << 17) | ((uint32_t)(TC_BM >> 4) << 24);
}

// Sixteen columns of a row through an activation (THA_ACT_*) and out as bf16: the branch on the activation is taken once per sixteen.
template <int ACT>
__device__ __forceinline__ void bf_act16_of(const uint32_t (&vg)[16], const uint32_t (&vu)[16], float limit, float alpha, __nv_bfloat16* o, long long ld, int n) {
#pragma unroll
  for (int j = 0; j < 16; j++) {
    if (j < n) hyb_store(o, hyb_act_value(ACT, __uint_as_float(vg[j]), __uint_as_float(vu[j]), limit, alpha));
    o += ld;
  }
}
template <bool GATED>
__device__ __forceinline__ void bf_act16(int act, const uint32_t (&vg)[16], const uint32_t (&vu)[16], float limit, float alpha, __nv_bfloat16* o,
                                         long long ld, int n) {
  if (!GATED) bf_act16_of<THA_ACT_RELU2>(vg, vu, limit, alpha, o, ld, n);
  else if (act == THA_ACT_SILU_GLU) bf_act16_of<THA_ACT_SILU_GLU>(vg, vu, limit, alpha, o, ld, n);
  else if (act == THA_ACT_GELU_TANH_GLU) bf_act16_of<THA_ACT_GELU_TANH_GLU>(vg, vu, limit, alpha, o, ld, n);
  else bf_act16_of<THA_ACT_GLU_CLAMPED>(vg, vu, limit, alpha, o, ld, n);
}

// BF_SWIGLU, BF_GATED (MT = 2): the two 128-row halves of a work item are the SAME rows of two matrices (mw0 = w1, mw1 = w3); the
// read-out combines the two accumulators of a row into silu(a) * c (run.cc:344-347 order) or a layer program's gated activation and
// stores it as bf16.  BF_UNGATED: the tiles of BF_PLAIN, an activation of the accumulator stored as bf16.
// A pair's tile has 128 columns: its two accumulators leave room for a second pair, so the read-out (an exponential and a division per
// element) runs behind the next item's products.  256 columns pull a quarter less through L2 but nothing hides their read-out: 4000 rows x
// [2 x 6144, 2048] 234 us against 154, 2825 x [2 x 11008, 4096] 499 against 385; two prompts of a 7B bf16 model 2.64 -> 2.59 ms.
template <int NT, int MT = 1, int READ = BF_PLAIN>
__global__ void __launch_bounds__(128 + 128 * MT, 1)
gemm_bf16_kernel(const __grid_constant__ CUtensorMap mw0, const __grid_constant__ CUtensorMap mw1,
                 const __grid_constant__ CUtensorMap mw2, const __grid_constant__ CUtensorMap mx, const BfP p) {
  using S = BfSmem<NT, MT>;
  constexpr int NBUF = S::NBUF;
  constexpr bool PAIR = READ == BF_SWIGLU || READ == BF_GATED;
  extern __shared__ unsigned char tc_smem_raw[];
  unsigned char* smem = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(tc_smem_raw) + 1023) & ~(uintptr_t)1023);
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + S::NST * S::STAGE);
  uint64_t* full = bars;                 // stage landed (W + X bytes)
  uint64_t* empty = full + S::NST;       // the MMAs that read the stage have completed
  uint64_t* accum = empty + S::NST;      // [2] accumulator buffer complete
  uint64_t* accfree = accum + 2;         // [2] ... and read out by the four epilogue warps
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(accfree + 2);
  int* abort_flag = reinterpret_cast<int*>(tmem_slot + 1);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  struct Item { int mat, row0, n0, kb0, nkb, wrow, xrow; };
  auto item_of = [&](int it) -> Item {
    Item w;
    const int z = it % p.splits;
    const int t = it / p.splits;
    int tile = t / p.ny;
    w.n0 = (t - tile * p.ny) * NT;
    w.mat = 0;
    while (w.mat + 1 < p.n_mats && tile >= p.tiles[w.mat]) { tile -= p.tiles[w.mat]; w.mat++; }
    w.row0 = tile * (PAIR ? TC_BM : TC_BM * MT);
    w.wrow = p.w_row[w.mat] + w.row0;   // where the tile lies in its tensor maps
    w.xrow = p.x_row[w.mat] + w.n0;
    w.kb0 = z * p.kblocks_per_split;
    w.nkb = p.kblocks_total - w.kb0;
    if (w.nkb > p.kblocks_per_split) w.nkb = p.kblocks_per_split;
    return w;
  };

  if (threadIdx.x == 0) {
    for (int s = 0; s < S::NST; s++) { tc_mbar_init(&full[s], 1); tc_mbar_init(&empty[s], 1); }
    for (int b = 0; b < 2; b++) { tc_mbar_init(&accum[b], 1); tc_mbar_init(&accfree[b], 4 * MT); }
    *abort_flag = 0;
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

  if (warp == 0) {
    // ===== TMA producer
    if (tc_elect()) {
      uint64_t pol_w;
      asm volatile("createpolicy.fractional.L2::evict_first.b64 %0, 1.0;" : "=l"(pol_w));
      const bool stream_w = p.ny == 1;            // every weight tile is read once: do not let it displace the activations in L2
      int gb = 0;
      bool ok = true, first = true;
      int sent = 0;
      auto load_w = [&](unsigned char* dst, const CUtensorMap* mw, int kcol, int row0, uint64_t* bar) {
        if (PAIR) {   // 128 rows of w1, then the same 128 rows of w3
          tc_tma_2d(dst, &mw0, kcol, row0, bar);
          tc_tma_2d(dst + TC_BM * 128, &mw1, kcol, row0, bar);
        } else if (stream_w) tc_tma_2d_hint(dst, mw, kcol, row0, bar, pol_w);
        else tc_tma_2d(dst, mw, kcol, row0, bar);
      };
      for (int it = blockIdx.x; it < p.n_items && ok; it += gridDim.x) {
        const Item w = item_of(it);
        const CUtensorMap* mw = (w.mat == 0 || p.stacked) ? &mw0 : (w.mat == 1 ? &mw1 : &mw2);
        int i = 0;
        if (first) {
          // weights never depend on the previous kernel: the first ring goes out before the dependency wait (the bytes may
          // land before the matching expect_tx -- the phase cannot complete until that arrival)
          const int pre = w.nkb < S::NST ? w.nkb : S::NST;
          for (; i < pre; i++) load_w(smem + i * S::STAGE, mw, (w.kb0 + i) * BF_BK, w.wrow, &full[i]);
          pdl_wait();
          for (int j = 0; j < pre; j++) {
            tc_mbar_expect_tx(&full[j], S::STAGE);
            tc_tma_2d(smem + j * S::STAGE + S::W_BYTES, &mx, (w.kb0 + j) * BF_BK, w.xrow, &full[j]);
          }
          first = false;
        }
        for (; i < w.nkb; i++) {
          const int g = gb + i, s = g % S::NST;
          if (g >= S::NST && !tc_mbar_wait(&empty[s], ((g / S::NST) & 1u) ^ 1u, abort_flag)) { ok = false; sent = g; break; }
          tc_mbar_expect_tx(&full[s], S::STAGE);
          load_w(smem + s * S::STAGE, mw, (w.kb0 + i) * BF_BK, w.wrow, &full[s]);
          tc_tma_2d(smem + s * S::STAGE + S::W_BYTES, &mx, (w.kb0 + i) * BF_BK, w.xrow, &full[s]);
        }
        gb += w.nkb;
      }
      if (!ok) tc_drain(full, S::NST, sent);
    }
  } else if (warp == 1) {
    // ===== MMA issuer
    if (tc_elect()) {
      constexpr uint32_t idesc = bf_idesc(NT);
      int gb = 0, n_it = 0;
      bool ok = true;
      for (int it = blockIdx.x; it < p.n_items && ok; it += gridDim.x, n_it++) {
        const Item w = item_of(it);
        const int buf = n_it % NBUF, use = n_it / NBUF;   // use-th time this buffer is filled
        if (use >= 1) {                            // the buffer's previous accumulator must have been read out
          if (!tc_mbar_wait(&accfree[buf], (unsigned)(use & 1) ^ 1u, abort_flag)) break;
          asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        }
        const uint32_t d = tmem_base + (uint32_t)(buf * MT * NT);
        for (int i = 0; i < w.nkb; i++) {
          const int g = gb + i, s = g % S::NST;
          if (!tc_mbar_wait(&full[s], (g / S::NST) & 1u, abort_flag)) { ok = false; break; }
          asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
          const uint64_t adesc = tc_smem_desc(tc_smem_u32(smem + s * S::STAGE));
          const uint64_t bdesc = tc_smem_desc(tc_smem_u32(smem + s * S::STAGE + S::W_BYTES));
#pragma unroll
          for (int k = 0; k < BF_BK / 16; k++)     // UMMA K = 16 bf16 = 32 bytes = 2 descriptor units
#pragma unroll
            for (int m = 0; m < MT; m++)           // the m-th 128 rows of the W stage: 16 KB = 1024 descriptor units further
              tc_mma_f16(d + (uint32_t)(m * NT), adesc + (uint64_t)(1024 * m + 2 * k), bdesc + (uint64_t)(2 * k), idesc, (uint32_t)((i | k) != 0));
          tc_commit(&empty[s]);
        }
        if (ok) tc_commit(&accum[buf]);
        gb += w.nkb;
      }
    }
  } else if (warp >= 4) {
    // ===== epilogue: thread = weight row of the tile (TMEM lane); warps 4-7 read the first 128 rows, 8-11 the second (MT = 2)
    const int q = warp & 3, mt = (warp - 4) >> 2;
    const int r = q * 32 + lane;
    pdl_trigger();
    pdl_wait();                                    // the column scales come from the previous kernel
    int n_it = 0;
    bool ok = true;
    for (int it = blockIdx.x; it < p.n_items; it += gridDim.x, n_it++) {
      const Item w = item_of(it);
      const int buf = n_it % NBUF, use = n_it / NBUF;
      if (ok) ok = tc_mbar_wait_warp(&accum[buf], (unsigned)(use & 1), abort_flag);
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      if (READ == BF_GATED || READ == BF_UNGATED) {
        // the row's accumulators (gate and up, or one) through the activation; warps 4-7 and 8-11 share the columns of a pair
        const int arow = w.row0 + (PAIR ? 0 : mt * TC_BM) + r;
        constexpr int C1 = PAIR ? NT / 2 : NT;
        const int c0 = PAIR ? mt * C1 : 0;
        const uint32_t ta = tmem_base + (uint32_t)(buf * MT * NT + (PAIR ? 0 : mt * NT)) + ((uint32_t)(q * 32) << 16);
        __nv_bfloat16* o = reinterpret_cast<__nv_bfloat16*>(p.act_out) + (size_t)(w.n0 + c0) * p.ld_act + arow;
        const int left = arow < p.M[0] ? p.N - w.n0 - c0 : 0;   // columns of this thread's row that are stored
        if (ok) {
#pragma unroll 1
          for (int c = 0; c < C1; c += 16, o += 16 * p.ld_act) {
            uint32_t vg[16], vu[16];
            tc_tmem_ld16(ta + (uint32_t)(c0 + c), vg);
            if (PAIR) tc_tmem_ld16(ta + (uint32_t)(NT + c0 + c), vu);
            asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
            bf_act16<PAIR>(p.act, vg, PAIR ? vu : vg, p.act_limit, p.act_alpha, o, p.ld_act, left - c);
          }
        }
        asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
        __syncwarp();
        if (lane == 0) tc_mbar_arrive(&accfree[buf]);
        continue;
      }
      if (READ == BF_SWIGLU) {
        // both accumulators of this thread's row; warps 4-7 take the first half of the columns, 8-11 the second
        const int srow = w.row0 + r;
        const uint32_t ta = tmem_base + (uint32_t)(buf * MT * NT) + ((uint32_t)(q * 32) << 16);
        const int cols = srow < p.M[0] ? p.N - w.n0 : 0;        // of this row that are stored; the loads are the whole warp's
        if (ok) {
          uint16_t* o = p.act_out + (size_t)(w.n0 + mt * (NT / 2)) * p.ld_act + srow;
#pragma unroll 1
          for (int c = mt * (NT / 2); c < (mt + 1) * (NT / 2); c += 16) {
            uint32_t va[16], vc[16];
            tc_tmem_ld16(ta + (uint32_t)c, va);
            tc_tmem_ld16(ta + (uint32_t)(NT + c), vc);
            asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
            for (int j = 0; j < 16; j++) {
              if (c + j < cols) {
                float h = __uint_as_float(va[j]);
                h *= (1.0f / (1.0f + expf(-h)));
                h *= __uint_as_float(vc[j]);
                const uint32_t u = __float_as_uint(h);   // round to nearest even, NaN stays NaN (step_bf16.cu f32_to_bf16)
                *o = ((u & 0x7FFFFFFFu) > 0x7F800000u) ? (uint16_t)((u >> 16) | 0x40u) : (uint16_t)((u + 0x7FFFu + ((u >> 16) & 1u)) >> 16);
              }
              o += p.ld_act;
            }
          }
        }
        asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
        __syncwarp();
        if (lane == 0) tc_mbar_arrive(&accfree[buf]);
        continue;
      }
      const int row = w.row0 + mt * TC_BM + r;
      const bool row_ok = row < p.M[w.mat];
      float* outz = p.out + (size_t)(it % p.splits) * p.zstride + p.out_off[w.mat] + row;
      const uint32_t tq = tmem_base + (uint32_t)(buf * MT * NT + mt * NT) + ((uint32_t)(q * 32) << 16);
      // whole tile inside the output: no per-element bounds checks, the store address advanced by one add per column
      // (the checked form costs ~25 instructions per element: gemm_tc.cu has the measurement)
      const bool full = row_ok && (w.n0 + NT <= p.N);
      const bool cs_vec = p.colscale && ((reinterpret_cast<uintptr_t>(p.colscale) & 15) == 0);
      if (ok) {
#pragma unroll 1
        for (int c = 0; c < NT; c += 32) {          // two 16-column loads in flight
          uint32_t v[32];
          tc_tmem_ld16(tq + (uint32_t)c, *reinterpret_cast<uint32_t(*)[16]>(v));
          if (NT > 16) tc_tmem_ld16(tq + (uint32_t)(c + 16), *reinterpret_cast<uint32_t(*)[16]>(v + 16));
          constexpr int NC = NT > 16 ? 32 : 16;
          float sc[NC];
          if (full && p.colscale) {
#pragma unroll
            for (int j = 0; j < NC; j += 4) {
              if (cs_vec) {
                const float4 t = __ldg(reinterpret_cast<const float4*>(p.colscale + w.n0 + c + j));
                sc[j] = t.x; sc[j + 1] = t.y; sc[j + 2] = t.z; sc[j + 3] = t.w;
              } else {
#pragma unroll
                for (int e = 0; e < 4; e++) sc[j + e] = __ldg(p.colscale + w.n0 + c + j + e);
              }
            }
          }
          asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
          if (full) {
            float* o = outz + (size_t)(w.n0 + c) * p.ldo;
#pragma unroll
            for (int j = 0; j < NC; j++) {
              float x = __uint_as_float(v[j]);
              if (p.colscale) x *= sc[j];
              *o = x;
              o += p.ldo;
            }
          } else {   // the last column tile, most prompts': 2000 rows x [2048, 2048] 30.1 -> 26.9 us, 4000 x [1024, 1024] 21.6 -> 18.7 against a multiply an address
            float* o = outz + (size_t)(w.n0 + c) * p.ldo;
            const int left = row_ok ? p.N - w.n0 - c : 0;
#pragma unroll
            for (int j = 0; j < NC; j++) {
              if (j < left) {
                float x = __uint_as_float(v[j]);
                if (p.colscale) x *= p.colscale[w.n0 + c + j];
                *o = x;
              }
              o += p.ldo;
            }
          }
        }
      }
      asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
      __syncwarp();
      if (lane == 0) tc_mbar_arrive(&accfree[buf]);
    }
  }
  __syncthreads();
  if (warp == 2) {
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(S::TMEM_COLS));
  }
  if (threadIdx.x == 0 && *abort_flag && p.error_flag) *((volatile int*)p.error_flag) = 1;
}

// ---- few output tiles: the K range of a tile dealt to a cluster ------------------------------------------------------------
// A product of a few rows with a matrix of a few thousand (decoding) has 8 to 100 tiles of 128 outputs: with a CTA per tile most SMs
// idle and the time is one CTA's walk over K.  Here the CTAs of a cluster take a share of a tile's K range each, leave their
// partial tiles in their own shared memory and sum each other's through distributed shared memory, ranks in ascending order
// (bit-reproducible; no partials in global memory, no counters).  Bound by the latency of one share: launch, first loads, MMA chain,
// exchange.  Cold weights, a launch behind the other, before -> now: [2 rows] x [1024 x 4608] 24.1 -> 7.5 us, [2048 x 6144] 30.9 -> 9.7,
// [3088 x 2048] 13.0 -> 7.1; [100 rows] x [2048 x 6144] 37.7 -> 14.9.  One tile per cluster, a share's k-blocks are all
// in flight where the ring holds them; two CTAs fit an SM.
template <int NT>
struct BfcSmem {
  static constexpr int W_BYTES = TC_BM * 128, X_BYTES = NT * 128, STAGE = W_BYTES + X_BYTES;
  static constexpr int NST = NT <= 32 ? 5 : (NT == 64 ? 4 : 3);
  static constexpr int TMEM_COLS = NT < 32 ? 32 : NT;
  static constexpr int TOTAL = NST * STAGE + 1024 + (2 * NST + 1) * 8 + 64;
  static_assert(NST * STAGE >= NT * TC_BM * 4, "the partial tile reuses the ring");
  static_assert(2 * (TOTAL + 1024) <= 228 * 1024, "two CTAs per SM");
};

template <int NT>
__global__ void __launch_bounds__(BF_THREADS)
gemm_bf16_cluster_kernel(const __grid_constant__ CUtensorMap mw0, const __grid_constant__ CUtensorMap mw1,
                         const __grid_constant__ CUtensorMap mw2, const __grid_constant__ CUtensorMap mx, const BfP p) {
  using S = BfcSmem<NT>;
  extern __shared__ unsigned char tc_smem_raw[];
  unsigned char* smem = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(tc_smem_raw) + 1023) & ~(uintptr_t)1023);
  uint64_t* full = reinterpret_cast<uint64_t*>(smem + S::NST * S::STAGE);   // stage landed
  uint64_t* empty = full + S::NST;                                          // the MMAs that read the stage have completed
  uint64_t* accum = empty + S::NST;                                         // this share's accumulator complete
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(accum + 1);
  int* abort_flag = reinterpret_cast<int*>(tmem_slot + 1);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int cl = p.splits, rank = (int)(blockIdx.x % cl);     // cluster = `cl` consecutive CTAs
  int tile = (int)(blockIdx.x / cl) / p.ny;
  const int n0 = ((int)(blockIdx.x / cl) - tile * p.ny) * NT;
  int mat = 0;
  while (mat + 1 < p.n_mats && tile >= p.tiles[mat]) { tile -= p.tiles[mat]; mat++; }
  const int row0 = tile * TC_BM;
  const int kb0 = rank * p.kblocks_per_split;
  const int nkb = max(0, min(p.kblocks_total - kb0, p.kblocks_per_split));

  if (threadIdx.x == 0) {
    for (int s = 0; s < S::NST; s++) { tc_mbar_init(&full[s], 1); tc_mbar_init(&empty[s], 1); }
    tc_mbar_init(accum, 1);
    *abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  }
  if (warp == 2) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(tc_smem_u32(tmem_slot)), "r"(S::TMEM_COLS));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::);
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem_d = *tmem_slot;

  if (warp == 0) {
    if (tc_elect()) {
      const CUtensorMap* mw = (mat == 0 || p.stacked) ? &mw0 : (mat == 1 ? &mw1 : &mw2);
      const int wrow = p.w_row[mat] + row0, xrow = p.x_row[mat] + n0;
      uint64_t pol_w;
      asm volatile("createpolicy.fractional.L2::evict_first.b64 %0, 1.0;" : "=l"(pol_w));
      auto load_w = [&](int i, int s) {
        if (p.ny == 1) tc_tma_2d_hint(smem + s * S::STAGE, mw, (kb0 + i) * BF_BK, wrow, &full[s], pol_w);
        else tc_tma_2d(smem + s * S::STAGE, mw, (kb0 + i) * BF_BK, wrow, &full[s]);
      };
      // the first ring of weights goes out ahead of the dependency wait (bytes may land before the matching expect_tx)
      const int pre = nkb < S::NST ? nkb : S::NST;
      for (int i = 0; i < pre; i++) load_w(i, i);
      pdl_wait();
      for (int i = 0; i < pre; i++) {
        tc_mbar_expect_tx(&full[i], S::STAGE);
        tc_tma_2d(smem + i * S::STAGE + S::W_BYTES, &mx, (kb0 + i) * BF_BK, xrow, &full[i]);
      }
      for (int i = pre; i < nkb; i++) {
        const int s = i % S::NST;
        if (!tc_mbar_wait(&empty[s], ((i / S::NST) & 1u) ^ 1u, abort_flag)) { tc_drain(full, S::NST, i); break; }
        tc_mbar_expect_tx(&full[s], S::STAGE);
        load_w(i, s);
        tc_tma_2d(smem + s * S::STAGE + S::W_BYTES, &mx, (kb0 + i) * BF_BK, xrow, &full[s]);
      }
    }
  } else if (warp == 1) {
    if (tc_elect()) {
      constexpr uint32_t idesc = bf_idesc(NT);
      bool ok = true;
      for (int i = 0; i < nkb; i++) {
        const int s = i % S::NST;
        if (!tc_mbar_wait(&full[s], (i / S::NST) & 1u, abort_flag)) { ok = false; break; }
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        const uint64_t adesc = tc_smem_desc(tc_smem_u32(smem + s * S::STAGE));
        const uint64_t bdesc = tc_smem_desc(tc_smem_u32(smem + s * S::STAGE + S::W_BYTES));
#pragma unroll
        for (int k = 0; k < BF_BK / 16; k++) tc_mma_f16(tmem_d, adesc + (uint64_t)(2 * k), bdesc + (uint64_t)(2 * k), idesc, (uint32_t)((i | k) != 0));
        tc_commit(&empty[s]);
      }
      if (ok && nkb > 0) tc_commit(accum);
    }
  }
  float* part = reinterpret_cast<float*>(smem);   // [NT][128], over the ring once its last MMA has read it
  if (warp >= 4) {
    const int r = (warp & 3) * 32 + lane;
    pdl_trigger();
    const bool ok = nkb > 0 && tc_mbar_wait(accum, 0u, abort_flag);
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
#pragma unroll 1
    for (int c = 0; c < NT; c += 16) {
      uint32_t v[16];
      if (ok) {
        tc_tmem_ld16(tmem_d + ((uint32_t)((warp & 3) * 32) << 16) + (uint32_t)c, v);
        asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
      }
#pragma unroll
      for (int j = 0; j < 16; j++) part[(c + j) * TC_BM + r] = ok ? __uint_as_float(v[j]) : 0.0f;
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  }
  __syncthreads();
  asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
  asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
  {
    // this rank's columns: rank, rank + cl, ... of the tile; half of the threads each take one at a time, a thread a row
    pdl_wait();   // returns at once (the producer waited): the column scales of the previous kernel are visible here
    const int r = threadIdx.x & (TC_BM - 1), row = row0 + r;
    const int n_cols = min(NT, p.N - n0);
    const uint32_t base = tc_smem_u32(part) + (uint32_t)r * 4u;
    for (int c = rank + cl * (int)(threadIdx.x >> 7); c < n_cols; c += 2 * cl) {
      float acc = 0.0f;
      for (int z = 0; z < cl; z++) {
        uint32_t a;
        float v;
        asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"(base + (uint32_t)(c * TC_BM * 4)), "r"(z));
        asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v) : "r"(a) : "memory");
        acc += v;
      }
      if (p.colscale) acc *= p.colscale[n0 + c];
      if (row < p.M[mat]) p.out[(size_t)(n0 + c) * p.ldo + p.out_off[mat] + row] = acc;
    }
  }
  asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");   // a CTA's shared memory stays until every rank has read it
  asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
  if (warp == 2) {
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_d), "r"(S::TMEM_COLS));
  }
  if (threadIdx.x == 0 && *abort_flag && p.error_flag) *((volatile int*)p.error_flag) = 1;
}

// ------------------------------------------------------------------ host side ----
bool gemm_bf16_ok(const BfArgs& a) {
  if (a.K % 8 || a.ldx % 8 || a.K < BF_BK || a.N < 1 || a.n_mats < 1 || a.n_mats > (a.stacked ? BF_MAX_MATS : 3) || !a.X || !a.out) return false;
  if (reinterpret_cast<uintptr_t>(a.X) & 15u) return false;
  for (int i = 0; i < a.n_mats; i++) {
    const uint16_t* w = a.W[a.stacked ? 0 : i];
    if (!w || (reinterpret_cast<uintptr_t>(w) & 15u) || a.M[i] < 1) return false;
  }
  return true;
}


template <int NT, int MT = 1, int READ = BF_PLAIN>
static int bf_launch_nt(cudaStream_t st, const CUtensorMap* mw, const CUtensorMap& mx, const BfP& p, dim3 grid, bool pdl) {
  using S = BfSmem<NT, MT>;
  auto k = gemm_bf16_kernel<NT, MT, READ>;
  THA_CUDA_OK(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, S::TOTAL));
  THA_CUDA_OK(launch(k, grid, dim3(128 + 128 * MT), (size_t)S::TOTAL, st, pdl, mw[0], mw[1], mw[2], mx, p));
  return THA_STATUS_SUCCESS;
}
// Output tile (128 mt weight rows x nt activation rows) of a product of `tiles` 128-row weight tiles with N activation rows: the one whose
// waves over the SMs cost least.  A wave of 256 x 256 / 128 x 256 / 128 x 128 / 128 x 64 tiles takes 50 / 28 / 20.5 / 19.5 us at K = 4096
// (small tiles pull more through L2 per product), so a large tile pays once it fills the SMs.  Measured, us, in that order: 2100 rows x
// [4096, 4096] 54 / 59 / 86 / 155; 2825 x [4096, 4096] 92 / 80 / 103 / 190; 2100 x [1024, 4608] 53 / 33 / 30 / 49; 700 x [2048, 2048] 35 / 25 / 19 / 26;
// 4000 x [12288, 4096] 313 / 312 / 409 / 763.
BfTile gemm_bf16_tile(int tiles, int N, int splits) {
  if (N <= 128) return {N <= 16 ? 16 : (N <= 32 ? 32 : (N <= 64 ? 64 : 128)), 1};
  static const struct { BfTile t; int cost; } form[4] = {{{256, 2}, 100}, {{256, 1}, 56}, {{128, 1}, 41}, {{64, 1}, 39}};
  BfTile best = form[0].t;
  long long least = 0;
  for (int i = 0; i < 4; i++) {
    const long long items = (long long)ceil_div(tiles, form[i].t.mt) * ceil_div(N, form[i].t.nt) * splits;
    const long long c = (items + 147) / 148 * form[i].cost;
    if (i == 0 || c < least) { least = c; best = form[i].t; }
  }
  return best;
}

template <int NT>
static cudaLaunchConfig_t bfc_config(cudaLaunchAttribute* attr, int grid, int cl, cudaStream_t st, bool pdl) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(grid); cfg.blockDim = dim3(BF_THREADS); cfg.dynamicSmemBytes = BfcSmem<NT>::TOTAL; cfg.stream = st;
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = cl; attr[0].val.clusterDim.y = 1; attr[0].val.clusterDim.z = 1;
  attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[1].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr; cfg.numAttrs = pdl ? 2 : 1;
  return cfg;
}
// CTAs per cluster for a product of `items` tiles over kb k-blocks, 1: a CTA per tile.  Two CTAs fit an SM (296 in all), but clusters
// have to fit a GPC's SMs together: from about 200 CTAs on some clusters wait for others to end.  Measured on both sides of the line,
// 2 rows, us at 1 / 2 / 4 / 8 ranks: [25 tiles, K 2048] 13.0 / 9.3 / 7.4 / 7.1 (200 CTAs of 8); [36, 1024] 8.7 / 7.2 / 6.5 / 9.5 (288);
// [49, 1024] 9.0 / 7.5 / 6.9 / 10.1; [96, 2048] 14.8 / 13.2 / 16.4 / 19.0; [250, 2048] 27.7 / 28.7 / 34.1 / 45.0.  A pair of CTAs does not pay
// for 128-column tiles (100 rows, [36, 1024]: 15.0 / 15.6 / 11.3; [96, 2048]: 21.6 / 22.9).
// Prompts (more than 128 rows, whose tile gemm_bf16_tile chose for a CTA each): four and eight ranks, from K = 4096 on.  us without / with:
// [1024 x 4608] 129 rows 18.9 / 12.6, 384 rows 18.8 / 15.2; [2048 x 6144] 129 rows 23.1 / 16.8; at K = 2048 about even ([1024 x 2048] 129 rows
// 12.4 / 10.7, 384 rows 11.0 / 12.7); at 1024 slower ([1024 x 1024] 256 rows 8.4 / 10.6); pairs slower throughout ([4096 x 4096] 129 rows
// 18.8 / 22.6, [3088 x 2048] 192 rows 12.6 / 16.6, [2048 x 6144] 256 rows 22.9 / 25.0).
static int bfc_ranks(int nt, int rows, int items, int kb) {
  if (rows > 128 && kb < 4096 / BF_BK) return 1;
  for (int cl = 8; cl > (nt == 128 || rows > 128 ? 2 : 1); cl >>= 1)
    if (kb >= 2 * cl && items * cl <= 200) return cl;
  return 1;
}
// Launches the cluster form where its rule takes it; *taken says whether it did.
template <int NT>
static int bfc_try(cudaStream_t st, const CUtensorMap* mw, const CUtensorMap& mx, BfP p, bool pdl, bool* taken) {
  const int cl = bfc_ranks(NT, p.N, p.n_items, p.kblocks_total);
  *taken = cl > 1;
  if (cl <= 1) return THA_STATUS_SUCCESS;
  p.splits = cl;
  p.kblocks_per_split = ceil_div(p.kblocks_total, cl);
  auto k = gemm_bf16_cluster_kernel<NT>;
  THA_CUDA_OK(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, BfcSmem<NT>::TOTAL));
  cudaLaunchAttribute attr[2];
  const cudaLaunchConfig_t cfg = bfc_config<NT>(attr, p.n_items * cl, cl, st, pdl);
  count_launch();
  THA_CUDA_OK(cudaLaunchKernelEx(&cfg, k, mw[0], mw[1], mw[2], mx, p));
  trace_launch(reinterpret_cast<const void*>(k), st);
  return THA_STATUS_SUCCESS;
}

static bool bf_act_pair(const BfArgs& a) { return a.ff_act == 0 || hyb_act_gated(a.ff_act - 1); }

// Where the activation in the read-out is the faster way.  us as product and activation / in one, by rows:
//   gated    [2 x 4608, 1024]  256: 12.5 / 16.5  400: 25.0 / 17.1  1000: 41 / 26  4000: 118 / 78
//            [2 x 6144, 2048]  256: 22.7 / 22.7  400: 41.3 / 32.9  1000: 76 / 43  4000: 258 / 154
//            [2 x 11008, 4096] 256: 57.6 / 63.6  400: 99.6 / 83.2  1000: 189 / 153  4000: 777 / 544
//   RELU2    [4608, 1024]  160: 12.5 / 8.8  256: 12.4 / 9.5  1000: 35 / 16.5  4000: 84 / 37
//            [11008, 4096]  160: 50 / 37  1000: 117 / 81  4000: 421 / 289
// expm1f outweighs the pass that it saves: XIELU [6144, 2048]  160: 19.5 / 20.6  1000: 55 / 59  4000: 140 / 162, so it keeps its own.
bool gemm_bf16_act_ok(const BfArgs& a) {
  if (!a.act_out || a.splits > 1 || a.stacked || a.colscale || a.ff_act == 1 + THA_ACT_XIELU) return false;
  if (!bf_act_pair(a)) return a.n_mats == 1 && a.N > 128;
  return a.n_mats == 2 && a.M[0] == a.M[1] && a.N >= (a.ff_act ? 257 : 512);
}

int gemm_bf16_launch(cudaStream_t st, const BfArgs& a, bool pdl) {
  if (!gemm_bf16_ok(a)) return THA_STATUS_INVALID_ARG;
  const bool act = a.act_out != nullptr, pair = act && bf_act_pair(a);
  if (act && !gemm_bf16_act_ok(a)) return THA_STATUS_NOT_SUPPORTED;
  int tiles128 = 0;
  for (int i = 0; i < a.n_mats; i++) tiles128 += ceil_div(a.M[i], TC_BM);
  const BfTile tile = pair ? BfTile{128, 1} : gemm_bf16_tile(tiles128, a.N, a.splits < 1 ? 1 : a.splits);
  const int NT = tile.nt, MT = tile.mt;   // pairs: 128-row boxes of each of the two matrices (the kernel itself runs MT = 2)
  CUtensorMap mw[3], mx;
  BfP p = {};
  int tiles = 0;
  p.n_mats = a.n_mats; p.stacked = a.stacked;
  int x_rows = a.N;
  if (a.stacked) {
    int w_rows = 0;
    for (int i = 0; i < a.n_mats; i++) {
      p.M[i] = a.M[i]; p.tiles[i] = ceil_div(a.M[i], TC_BM * MT); p.out_off[i] = a.out_off[i];
      p.w_row[i] = a.w_row[i]; p.x_row[i] = a.x_row[i];
      w_rows = max(w_rows, a.w_row[i] + a.M[i]);
      x_rows = max(x_rows, a.x_row[i] + a.N);
      tiles += p.tiles[i];
    }
    THA_TRY_RC(tc_map(a.W[0], w_rows, a.K, a.K, TC_BM * MT, &mw[0], 2));
    mw[1] = mw[2] = mw[0];
  }
  for (int i = 0; i < 3 && !a.stacked; i++) {
    if (i < a.n_mats) {
      THA_TRY_RC(tc_map(a.W[i], a.M[i], a.K, a.K, TC_BM * MT, &mw[i], 2));
      p.M[i] = a.M[i]; p.tiles[i] = ceil_div(a.M[i], TC_BM * MT); p.out_off[i] = a.out_off[i];
    } else {
      mw[i] = mw[0];
    }
    tiles += p.tiles[i];
  }
  if (pair) { tiles = p.tiles[0]; p.tiles[1] = 0; p.n_mats = 1; }   // an item = a pair of tiles
  p.act_out = a.act_out; p.ld_act = a.ld_act;
  p.act = a.ff_act - 1; p.act_limit = a.act_limit; p.act_alpha = a.act_alpha;
  THA_TRY_RC(tc_map(a.X, x_rows, a.K, a.ldx, NT, &mx, 2));
  p.K = a.K; p.N = a.N;
  p.kblocks_total = ceil_div(a.K, BF_BK);
  const int splits = a.splits < 1 ? 1 : a.splits;
  p.kblocks_per_split = ceil_div(p.kblocks_total, splits);
  if (ceil_div(p.kblocks_total, p.kblocks_per_split) != splits) return THA_STATUS_INVALID_ARG;
  p.out = a.out; p.ldo = a.ldo; p.zstride = a.zstride; p.colscale = a.colscale;
  THA_TRY_RC(gemm_tc_init(&p.error_flag));
  p.ny = ceil_div(a.N, NT);
  p.splits = splits;
  p.n_items = tiles * p.ny * splits;
  if (splits == 1 && !act && NT <= 128) {   // callers that split K themselves sum the partials in a kernel of theirs
    bool taken = false;
    int rc = THA_STATUS_SUCCESS;
    switch (NT) {
      case 16: rc = bfc_try<16>(st, mw, mx, p, pdl, &taken); break;
      case 32: rc = bfc_try<32>(st, mw, mx, p, pdl, &taken); break;
      case 64: rc = bfc_try<64>(st, mw, mx, p, pdl, &taken); break;
      default: rc = bfc_try<128>(st, mw, mx, p, pdl, &taken);
    }
    if (taken || rc != THA_STATUS_SUCCESS) return rc;
  }
  int dev = 0, sms = 148;
  if (cudaGetDevice(&dev) == cudaSuccess) cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  dim3 grid(p.n_items < sms ? p.n_items : sms, 1, 1);
  switch (NT) {
    case 16: return bf_launch_nt<16>(st, mw, mx, p, grid, pdl);
    case 32: return bf_launch_nt<32>(st, mw, mx, p, grid, pdl);
    case 64: return act ? bf_launch_nt<64, 1, BF_UNGATED>(st, mw, mx, p, grid, pdl) : bf_launch_nt<64>(st, mw, mx, p, grid, pdl);
    case 128:
      if (pair) return a.ff_act ? bf_launch_nt<128, 2, BF_GATED>(st, mw, mx, p, grid, pdl) : bf_launch_nt<128, 2, BF_SWIGLU>(st, mw, mx, p, grid, pdl);
      return act ? bf_launch_nt<128, 1, BF_UNGATED>(st, mw, mx, p, grid, pdl) : bf_launch_nt<128>(st, mw, mx, p, grid, pdl);
    default:
      if (MT == 2) return act ? bf_launch_nt<256, 2, BF_UNGATED>(st, mw, mx, p, grid, pdl) : bf_launch_nt<256, 2>(st, mw, mx, p, grid, pdl);
      return act ? bf_launch_nt<256, 1, BF_UNGATED>(st, mw, mx, p, grid, pdl) : bf_launch_nt<256>(st, mw, mx, p, grid, pdl);
  }
}

}  // namespace tha

using namespace tha;

// C-ABI: out[n*ldo + row] = sum_k W[row,k] X[n,k], W and X bf16 (raw 16-bit patterns), fp32 out
extern "C" int tha_gemm_bf16(void* stream, float* out, long long ldo, const uint16_t* W, int M, int K, const uint16_t* X, int N,
                             long long ldx) {
  if (!out || !W || !X || M < 1 || N < 1 || K < 1) return THA_STATUS_INVALID_ARG;
  BfArgs a = {};
  a.n_mats = 1; a.W[0] = W; a.M[0] = M; a.out_off[0] = 0; a.K = K; a.X = X; a.N = N; a.ldx = ldx;
  a.out = out; a.ldo = ldo; a.zstride = 0; a.splits = 1; a.colscale = nullptr;
  if (!gemm_bf16_ok(a)) return THA_STATUS_NOT_SUPPORTED;
  return gemm_bf16_launch((cudaStream_t)stream, a, false);
}
