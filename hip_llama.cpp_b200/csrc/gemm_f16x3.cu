// fp32 weight matmul of prompts on the tensor cores: three fp16 products of operands split in two.
//
//   out[n, row] = sum_k W[row, k] * X[n, k]          W: [M, K] row-major fp32, X: [N, K] as two fp16 planes and a power of two a row
//
// A value times a power of two of its row is hi + lo 2^-11 (split_f16.cuh): 22 bits of significand, as tf32 hi and lo keep, at twice the MMA rate and half the
// bytes.  The largest value of a row of X is brought to [2^14, 2^15): values down to 2^-28 of it keep their 22 bits, none loses more than 2^-50 of it.  The scale of
// a weight row comes from its first values: the largest of up to 128 (of a share of K) is brought to [2^7, 2^8), which leaves a factor of 256 above it; values down to 2^-21 of
// it keep their 22 bits, none loses more than 2^-43 of it.  A row that goes further up than that, or whose first values are all zero, shows as an infinity in hi: the CTA pair
// then goes over its items once more with scales of the whole rows.  Whi.Xhi and the two corrections have accumulators of their own, so that the large
// sum takes K / 16 additions (3xTF32: K / 8); the corrections join it in the read-out, times 2^-11.
//
// A pair of CTAs (cta_group::2) takes 256 weight rows x 128 activation rows: each has 128 of the weight rows, in TMEM, and 64 of the activation rows, in shared
// memory, that both halves of the MMA read.  Bound by the tensor pipe under the power limit (73 % of its cycles active at 1024 rows x 12288 x 4096) and by the last, partly
// filled round over the 74 pairs (51 % at 1936 rows of 768, 4096 outputs); the tf32 kernel was bound by what reaches shared memory through L2: per 64 values of K a CTA loads
// 32 KB of weights and 16 KB of activations for 768 cycles of MMAs, there 32 + 64 KB for 1536 (and took 2100).  The kernel by itself, 1024 rows x 22016 x 4096: 675 us with
// 3xTF32, 472 with this, 400 for three products at the sustained cuBLAS bf16 rate; 4096 x 11008: 364, 238 (200); 1936 rows of 768, 4096 outputs: 58, 43 (26).
// The MMAs sum up runs of 1024 values of K, the read-out adds the runs in its registers: the tensor core's sum loses up to a unit in the last place with every
// addition.  Relative error at K = 4096: 9.6e-6 with 3xTF32, 4.9e-6 with one run, 1.25e-6 with runs of 1024 (6.5e-7 of 512; 3 and 7 % more time than one run).
// Announcements across the pair carry no generic memory, so no fence: with release and acquire at cluster scope the same products took 418 us in place of 267.
//   warp 0      TMA producer of W (weights: ahead of griddepcontrol.wait)
//   warp 1      rank 0: MMA issuer of the pair; rank 1: tells it that a stage of X has landed
//   warp 2      TMEM allocation
//   warp 3      TMA producer of X
//   warps 4-11  converters: two groups of four, k-blocks of 64 in turn; thread = weight row: 64 floats -> 32 + 32 TMEM columns
//   warps 12-19 read-out: thread = weight row x 64 activation rows.  The corrections leave TMEM first, since the next item's MMAs write
//               them again; the main sum has two buffers.
#include <cuda.h>

#include "common.cuh"
#include "gemm_tc.h"
#include "split_f16.cuh"
#include "tc_common.cuh"

namespace tha {

constexpr int X3_THREADS = 640;
constexpr int X3_BOUND = 768;            // 80 registers a thread at launch, 51200 a block, so that blocks of the row kernels around it fit beside it; then
                                         // 128 x 48 + 256 x 72 + 256 x 104, the same
constexpr int X3_BK = 64;                // values per k-block
constexpr int X3_NT = 128;               // activation rows of a pair
constexpr int X3_CONV_WARPS = 8;
constexpr int X3_RUN = 16;               // k-blocks that the MMAs sum up; runs are summed in the read-out's registers

struct X3P {
  const float* W[3]; int M[3]; int tiles[3]; int out_off[3];
  int K, N, ny, kblocks_total, kblocks_per_split;
  float* out; long long ldo; long long zstride;
  const float* colscale;
  int* error_flag;
  int splits, n_items;
};

struct X3Smem {
  static constexpr int W_STAGE = 2 * TC_BM * 128;       // two boxes of 32 floats
  static constexpr int X_PLANE = (X3_NT / 2) * 128;     // 64 rows of 64 halves
  static constexpr int X_STAGE = 2 * X_PLANE;           // hi | lo
  static constexpr int SW = 4, SX = 5;
  static constexpr int NBARS = 2 * SW + 3 * SX + 2 + 2 + 2 + 2 + 1 + 4 + 4 + 1;
  static constexpr int TOTAL = SW * W_STAGE + SX * X_STAGE + 1024 + NBARS * 8 + 64;
  // TMEM columns: main sum 0 | corrections | main sum 1 | two operand slots of 32 (hi) + 32 (lo)
  static constexpr int COL_CORR = 128, COL_MAIN1 = 256, COL_A = 384;
  static_assert(TOTAL <= TC_SMEM_LIMIT, "shared memory overflow");
};

__device__ __forceinline__ void x3_arrive_leader(uint64_t* bar) {   // the same barrier of the pair's rank 0.  What it announces is TMEM and TMA data, never generic memory of this thread
  uint32_t a;
  asm volatile("mapa.shared::cluster.u32 %0, %1, 0;" : "=r"(a) : "r"(tc_smem_u32(bar)));
  asm volatile("mbarrier.arrive.shared::cluster.b64 _, [%0];" ::"r"(a) : "memory");
}
__device__ __forceinline__ void x3_commit(uint64_t* bar) {   // to both CTAs
  asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;" ::"r"(tc_smem_u32(bar)), "h"((uint16_t)3) : "memory");
}
// kind::f16 with fp16 operands, fp32 accumulate, M = 256 over the pair, N = 128
constexpr uint32_t X3_IDESC = (1u << 4) | ((uint32_t)(X3_NT >> 3) << 17) | ((uint32_t)(256 >> 4) << 24);
__device__ __forceinline__ void x3_mma(uint32_t tmem_d, uint32_t tmem_a, uint64_t bdesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::2.kind::f16 [%0], [%1], %2, %3, p;\n\t}"
      ::"r"(tmem_d), "r"(tmem_a), "l"(bdesc), "r"(X3_IDESC), "r"(accumulate) : "memory");
}
__device__ __forceinline__ void x3_tmem_st16(uint32_t taddr, const uint32_t (&v)[16]) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16};"
      ::"r"(taddr), "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7]), "r"(v[8]), "r"(v[9]),
        "r"(v[10]), "r"(v[11]), "r"(v[12]), "r"(v[13]), "r"(v[14]), "r"(v[15]) : "memory");
}
constexpr int X3_SCALE_MOST = 115;       // powers of two of a row's scale at most

__global__ void __launch_bounds__(X3_BOUND, 1)
gemm_f16x3_kernel(const __grid_constant__ CUtensorMap mw0, const __grid_constant__ CUtensorMap mw1, const __grid_constant__ CUtensorMap mw2,
                  const __grid_constant__ CUtensorMap mxh, const __grid_constant__ CUtensorMap mxl, const __grid_constant__ X3P p) {
  using S = X3Smem;
  extern __shared__ unsigned char tc_smem_raw[];
  unsigned char* smem = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(tc_smem_raw) + 1023) & ~(uintptr_t)1023);
  unsigned char* wring = smem;
  unsigned char* xring = smem + S::SW * S::W_STAGE;
  uint64_t* wfull = reinterpret_cast<uint64_t*>(xring + S::SX * S::X_STAGE);   // W stage landed
  uint64_t* wfree = wfull + S::SW;       // ... and converted
  uint64_t* xfull = wfree + S::SW;       // X stage landed
  uint64_t* xpeer = xfull + S::SX;       // rank 0: ... in rank 1
  uint64_t* xempty = xpeer + S::SX;      // the MMAs that read it have completed
  uint64_t* aready = xempty + S::SX;     // [2] rank 0: operand slot filled in both CTAs
  uint64_t* aempty = aready + 2;         // [2] the MMAs that read it have completed
  uint64_t* accum = aempty + 2;          // [2] sums of an item complete
  uint64_t* mainfree = accum + 2;        // [2] rank 0: main sum read out in both CTAs
  uint64_t* corrfree = mainfree + 2;     // rank 0: corrections read out in both CTAs
  uint64_t* rowready = corrfree + 1;     // [4] scales of the weight rows of an item
  uint64_t* rowfree = rowready + 4;      // [4] ... and taken by the read-out
  uint64_t* mmadone = rowfree + 4;       // all MMAs complete
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(mmadone + 1);
  int* abort_flag = reinterpret_cast<int*>(tmem_slot + 1);
  int* bad_rows = abort_flag + 1;        // a weight row of this CTA went beyond the scale of its first values
  __shared__ float smax[4][2][TC_BM];    // largest of the first values of a weight row, by converter group; item mod 4
  __shared__ float rowf[4][TC_BM];       // inverse scale of a weight row

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int rank = blockIdx.x & 1, pair = blockIdx.x >> 1, n_pairs = gridDim.x >> 1;
  struct Item { int mat, row0, n0, kb0, nkb; };
  auto item_of = [&](int it) -> Item {
    Item w;
    const int z = it % p.splits, t = it / p.splits;
    int tile = t / p.ny;
    w.n0 = (t - tile * p.ny) * X3_NT;
    w.mat = 0;
    while (w.mat < 2 && tile >= p.tiles[w.mat]) { tile -= p.tiles[w.mat]; w.mat++; }
    w.row0 = tile * 2 * TC_BM + rank * TC_BM;
    w.kb0 = z * p.kblocks_per_split;
    w.nkb = min(p.kblocks_total - w.kb0, p.kblocks_per_split);
    return w;
  };

  if (threadIdx.x == 0) {
    for (int s = 0; s < S::SW; s++) { tc_mbar_init(&wfull[s], 1); tc_mbar_init(&wfree[s], 4); }
    for (int s = 0; s < S::SX; s++) { tc_mbar_init(&xfull[s], 1); tc_mbar_init(&xpeer[s], 1); tc_mbar_init(&xempty[s], 1); }
    for (int s = 0; s < 2; s++) { tc_mbar_init(&aready[s], 8); tc_mbar_init(&aempty[s], 1); tc_mbar_init(&accum[s], 1); tc_mbar_init(&mainfree[s], 16); }
    tc_mbar_init(corrfree, 16);
    tc_mbar_init(mmadone, 1);
    for (int s = 0; s < 4; s++) { tc_mbar_init(&rowready[s], 4); tc_mbar_init(&rowfree[s], 8); }
    *abort_flag = 0;
    *bad_rows = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  }
  if (warp == 0 && lane == 0) {
    asm volatile("prefetch.tensormap [%0];" ::"l"(&mw0) : "memory");
    if (p.tiles[1]) asm volatile("prefetch.tensormap [%0];" ::"l"(&mw1) : "memory");
    if (p.tiles[2]) asm volatile("prefetch.tensormap [%0];" ::"l"(&mw2) : "memory");
    asm volatile("prefetch.tensormap [%0];" ::"l"(&mxh) : "memory");
    asm volatile("prefetch.tensormap [%0];" ::"l"(&mxl) : "memory");
  }
  if (warp == 2) {
    asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(tc_smem_u32(tmem_slot)), "r"(512));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::);
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");   // both CTAs' barriers are there
  asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem = *tmem_slot;

  int gb = 0, n_it = 0, n_run = 0;      // k-blocks, items and runs so far, of both passes
  bool ok = true;
  int sent = -1;                        // stages that a producer has asked for, where it has given up
  // The end of a pass: whether there is another one, the same answer in both CTAs.  Every thread comes here, whatever became of its waits, and each of these is
  // bounded: so are the two CTAs' waits for each other.
  auto again = [&]() -> bool {
    __syncwarp();
    __syncthreads();
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
    uint32_t a;
    int peer;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"(tc_smem_u32(bad_rows)), "r"(rank ^ 1));
    asm volatile("ld.shared::cluster.s32 %0, [%1];" : "=r"(peer) : "r"(a) : "memory");
    return (peer | *bad_rows) != 0;
  };
  if (warp < 4) {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 48;");
    for (int pass = 0; pass < 2; pass++) {
      if (warp == 0) {
        if (tc_elect()) {
          for (int it = pair; it < p.n_items && ok; it += n_pairs) {
            const Item w = item_of(it);
            const CUtensorMap* mw = w.mat == 0 ? &mw0 : (w.mat == 1 ? &mw1 : &mw2);
            for (int i = 0; i < w.nkb; i++) {
              const int g = gb + i, s = g % S::SW;
              if (g >= S::SW && !tc_mbar_wait(&wfree[s], ((g / S::SW) & 1u) ^ 1u, abort_flag)) { ok = false; sent = g; break; }
              tc_mbar_expect_tx(&wfull[s], S::W_STAGE);
              unsigned char* dst = wring + s * S::W_STAGE;
              tc_tma_2d(dst, mw, (w.kb0 + i) * X3_BK, w.row0, &wfull[s]);
              tc_tma_2d(dst + TC_BM * 128, mw, (w.kb0 + i) * X3_BK + 32, w.row0, &wfull[s]);
            }
            gb += w.nkb;
          }
        }
      } else if (warp == 3) {
        if (tc_elect()) {
          pdl_wait();
          for (int it = pair; it < p.n_items && ok; it += n_pairs) {
            const Item w = item_of(it);
            for (int i = 0; i < w.nkb; i++) {
              const int g = gb + i, s = g % S::SX;
              if (g >= S::SX && !tc_mbar_wait(&xempty[s], ((g / S::SX) & 1u) ^ 1u, abort_flag)) { ok = false; sent = g; break; }
              tc_mbar_expect_tx(&xfull[s], S::X_STAGE);
              unsigned char* dst = xring + s * S::X_STAGE;
              tc_tma_2d(dst, &mxh, (w.kb0 + i) * X3_BK, w.n0 + rank * (X3_NT / 2), &xfull[s]);
              tc_tma_2d(dst + S::X_PLANE, &mxl, (w.kb0 + i) * X3_BK, w.n0 + rank * (X3_NT / 2), &xfull[s]);
            }
            gb += w.nkb;
          }
        }
      } else if (warp == 1) {
        if (tc_elect()) {
          for (int it = pair; it < p.n_items && ok; it += n_pairs, n_it++) {
            const Item w = item_of(it);
            if (rank) {
              for (int i = 0; i < w.nkb; i++) {
                const int g = gb + i, s = g % S::SX;
                if (!tc_mbar_wait(&xfull[s], (g / S::SX) & 1u, abort_flag)) { ok = false; break; }
                x3_arrive_leader(&xpeer[s]);
              }
              gb += w.nkb;
              continue;
            }
            for (int i0 = 0; i0 < w.nkb && ok; i0 += X3_RUN, n_run++) {
              const int buf = n_run & 1, use = n_run >> 1;
              if (use >= 1 && !tc_mbar_wait(&mainfree[buf], (unsigned)(use & 1) ^ 1u, abort_flag)) { ok = false; break; }
              if (n_run >= 1 && !tc_mbar_wait(corrfree, (unsigned)(n_run - 1) & 1u, abort_flag)) { ok = false; break; }
              const uint32_t d = tmem + (uint32_t)(buf ? S::COL_MAIN1 : 0), dc = tmem + S::COL_CORR;
              const int i1 = min(i0 + X3_RUN, w.nkb);
              for (int i = i0; i < i1; i++) {
                const int g = gb + i, s = g % S::SX, sa = g & 1;
                if (!tc_mbar_wait(&xfull[s], (g / S::SX) & 1u, abort_flag) || !tc_mbar_wait(&xpeer[s], (g / S::SX) & 1u, abort_flag) ||
                    !tc_mbar_wait(&aready[sa], (g >> 1) & 1u, abort_flag)) { ok = false; break; }
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                const uint64_t xh = tc_smem_desc(tc_smem_u32(xring + s * S::X_STAGE)), xl = xh + (uint64_t)(S::X_PLANE >> 4);
                const uint32_t ah = tmem + S::COL_A + sa * 64, al = ah + 32;
#pragma unroll
                for (int k = 0; k < X3_BK / 16; k++) {   // K = 16: 8 TMEM columns of A, 32 bytes (2 descriptor units) of B
                  x3_mma(dc, al + 8 * k, xh + (uint64_t)(2 * k), (uint32_t)((i - i0 | k) != 0));
                  x3_mma(dc, ah + 8 * k, xl + (uint64_t)(2 * k), 1u);
                  x3_mma(d, ah + 8 * k, xh + (uint64_t)(2 * k), (uint32_t)((i - i0 | k) != 0));
                }
                x3_commit(&aempty[sa]);
                x3_commit(&xempty[s]);
              }
              if (ok) x3_commit(&accum[buf]);
            }
            gb += w.nkb;
          }
        }
      }
      if (!again()) break;
    }
    if (*((volatile int*)abort_flag)) {                // copies and MMAs end ahead of the blocks
      if (warp == 0 && tc_elect()) tc_drain(wfull, S::SW, sent < 0 ? gb : sent);
      if (warp == 3 && tc_elect()) tc_drain(xfull, S::SX, sent < 0 ? gb : sent);
      if (warp == 1 && rank == 0 && tc_elect()) {
        x3_commit(mmadone);
        tc_drain(mmadone, 1, 1);
      }
    }
    __syncwarp();
  } else if (warp < 4 + X3_CONV_WARPS) {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 72;");
    for (int pass = 0; pass < 2; pass++) {
      // ===== converters: every thread takes part in every item's exchange of maxima, whatever became of its waits
      const int q = warp & 3, r = q * 32 + lane, grp = (warp >> 2) - 1;
      for (int it = pair; it < p.n_items; it += n_pairs, n_it++) {
        const Item w = item_of(it);
        const int i0 = (grp ^ gb) & 1, par = n_it & 3;
        float m = 0.0f;
        if (pass == 0) {
          if (i0 < w.nkb) {
            const int sw = (gb + i0) % S::SW;
            if (ok) ok = tc_mbar_wait_warp(&wfull[sw], ((gb + i0) / S::SW) & 1u, abort_flag);
            if (ok) {
              const unsigned char* wrow = wring + sw * S::W_STAGE + r * 128;
#pragma unroll
              for (int j = 0; j < 16; j++) {
                const float4 v = *reinterpret_cast<const float4*>(wrow + (j >> 3) * (TC_BM * 128) + (((j & 7) ^ (r & 7)) << 4));
                m = fmaxf(m, fmaxf(fmaxf(fabsf(v.x), fabsf(v.y)), fmaxf(fabsf(v.z), fabsf(v.w))));
              }
            }
          }
        } else if (w.row0 + r < p.M[w.mat]) {        // the item's share of the whole row
          const float* wr = p.W[w.mat] + (size_t)(w.row0 + r) * p.K;
          const int end = min(p.K, (w.kb0 + w.nkb) * X3_BK);
          for (int k = w.kb0 * X3_BK + 4 * grp; k < end; k += 8) {
            const float4 v = *reinterpret_cast<const float4*>(wr + k);
            m = fmaxf(m, fmaxf(fmaxf(fabsf(v.x), fabsf(v.y)), fmaxf(fabsf(v.z), fabsf(v.w))));
          }
        }
        smax[par][grp][r] = m;
        asm volatile("bar.sync 1, 256;" ::: "memory");
        float inverse;
        const float sc = split_scale<X3_SCALE_MOST>(fmaxf(smax[par][0][r], smax[par][1][r]), pass ? 14 : 7, &inverse);
        if (grp == 0) {
          // what the MMAs have completed says nothing of the read-out's last step: with a k-block an item these warps are four items ahead of it
          if (n_it >= 4 && ok) ok = tc_mbar_wait_warp(&rowfree[par], (unsigned)((n_it >> 2) & 1) ^ 1u, abort_flag);
          rowf[par][r] = inverse;
          __syncwarp();
          if (lane == 0) tc_mbar_arrive(&rowready[par]);
        }
        __half2 top = __half2half2(__ushort_as_half(0));
        for (int i = i0; i < w.nkb && ok; i += 2) {
          const int g = gb + i, sw = g % S::SW, sa = g & 1;
          ok = tc_mbar_wait_warp(&wfull[sw], (g / S::SW) & 1u, abort_flag);
          const uint32_t ta = tmem + S::COL_A + sa * 64 + ((uint32_t)(q * 32) << 16);
#pragma unroll
          for (int half = 0; half < 2; half++) {
            uint32_t hi[16], lo[16];
            const unsigned char* wrow = wring + sw * S::W_STAGE + half * (TC_BM * 128) + r * 128;
#pragma unroll
            for (int j = 0; j < 8; j++) {            // logical 16-byte chunk j lives at j ^ (row & 7) (SWIZZLE_128B)
              const float4 v = *reinterpret_cast<const float4*>(wrow + ((j ^ (r & 7)) << 4));
              split_f16x2(make_float2(v.x, v.y), sc, hi[2 * j], lo[2 * j]);
              split_f16x2(make_float2(v.z, v.w), sc, hi[2 * j + 1], lo[2 * j + 1]);
              top = __hmax2(top, __hmax2(__habs2(*reinterpret_cast<__half2*>(&hi[2 * j])), __habs2(*reinterpret_cast<__half2*>(&hi[2 * j + 1]))));
            }
            if (half == 0) {
              if (g >= 2 && ok) ok = tc_mbar_wait_warp(&aempty[sa], ((g >> 1) & 1u) ^ 1u, abort_flag);
              asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            }
            x3_tmem_st16(ta + (uint32_t)(16 * half), hi);
            x3_tmem_st16(ta + (uint32_t)(32 + 16 * half), lo);
          }
          __syncwarp();
          if (lane == 0) tc_mbar_arrive(&wfree[sw]);  // every value has been read and converted
          asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
          asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
          __syncwarp();
          if (lane == 0) x3_arrive_leader(&aready[sa]);
        }
        if (pass == 0 && (__hisinf(__low2half(top)) || __hisinf(__high2half(top)))) *bad_rows = 1;
        gb += w.nkb;
      }
      if (!again()) break;
    }
  } else {
    asm volatile("setmaxnreg.inc.sync.aligned.u32 104;");
    for (int pass = 0; pass < 2; pass++) {
      const int q = warp & 3, r = q * 32 + lane, c0 = (X3_NT / 2) * ((warp >> 2) - 1 - X3_CONV_WARPS / 4);
      pdl_trigger();
      pdl_wait();                                    // the column scales come from the previous kernel
      for (int it = pair; it < p.n_items; it += n_pairs, n_it++) {
        const Item w = item_of(it);
        const int par = n_it & 3;
        const uint32_t lanes = (uint32_t)(q * 32) << 16;
        float sum[X3_NT / 2];
#pragma unroll
        for (int j = 0; j < X3_NT / 2; j++) sum[j] = 0.0f;
        for (int i0 = 0; i0 < w.nkb; i0 += X3_RUN, n_run++) {
          const int buf = n_run & 1;
          if (ok) ok = tc_mbar_wait_warp(&accum[buf], (unsigned)(n_run >> 1) & 1u, abort_flag);
          asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
#pragma unroll
          for (int part = 0; part < 2; part++) {     // corrections, then the main sum
            const uint32_t tm = tmem + lanes + (uint32_t)(c0 + (part == 0 ? S::COL_CORR : (buf ? S::COL_MAIN1 : 0)));
#pragma unroll
            for (int c = 0; c < X3_NT / 2; c += 16) {
              uint32_t v[16];
              tc_tmem_ld16(tm + (uint32_t)c, v);
              asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
              for (int j = 0; j < 16; j++) sum[c + j] = part == 0 ? fmaf(__uint_as_float(v[j]), SPLIT_DOWN, sum[c + j]) : sum[c + j] + __uint_as_float(v[j]);
            }
            asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
            __syncwarp();
            if (lane == 0) x3_arrive_leader(part == 0 ? corrfree : &mainfree[buf]);
          }
        }
        if (ok) ok = tc_mbar_wait_warp(&rowready[par], (unsigned)(n_it >> 2) & 1u, abort_flag);
        const float rf = rowf[par][r];
        __syncwarp();
        if (lane == 0) tc_mbar_arrive(&rowfree[par]);
        const int row = w.row0 + r;
        if (!ok || row >= p.M[w.mat]) continue;
        float* o = p.out + (size_t)(it % p.splits) * p.zstride + p.out_off[w.mat] + row + (size_t)(w.n0 + c0) * p.ldo;
        const int n = w.n0 + c0;
        if (n + X3_NT / 2 <= p.N) {
#pragma unroll
          for (int j = 0; j < X3_NT / 2; j += 4) {
            const float4 s4 = *reinterpret_cast<const float4*>(p.colscale + n + j);
            const float sc[4] = {s4.x, s4.y, s4.z, s4.w};
#pragma unroll
            for (int e = 0; e < 4; e++) {
              *o = (sum[j + e] * rf) * sc[e];
              o += p.ldo;
            }
          }
        } else {
#pragma unroll
          for (int j = 0; j < X3_NT / 2; j++)
            if (n + j < p.N) {
              *o = (sum[j] * rf) * p.colscale[n + j];
              o += p.ldo;
            }
        }
      }
      if (!again()) break;
    }
  }
  asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");   // a CTA's barriers and flags stay until both are done
  asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
  if (warp == 2) {
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512));
  }
  if (threadIdx.x == 0 && *abort_flag && p.error_flag) *((volatile int*)p.error_flag) = 1;
}

// ---- rows -> two fp16 planes and the scale that takes a product back ---------------------------------------------------------
// Sum of s and maximum of m over the block (up to 1024 threads); red: 66 floats
__device__ __forceinline__ void x3_block_sum_max(float& s, float& m, float* red) {
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, nw = (blockDim.x + 31) >> 5;
  s = warp_sum(s);
  m = warp_max(m);
  if (lane == 0) { red[wid] = s; red[33 + wid] = m; }
  __syncthreads();
  s = warp_sum(lane < nw ? red[lane] : 0.0f);
  m = warp_max(lane < nw ? red[33 + lane] : 0.0f);
}
__device__ __forceinline__ float x3_abs_max(float4 v, float m) { return fmaxf(m, fmaxf(fmaxf(fabsf(v.x), fabsf(v.y)), fmaxf(fabsf(v.z), fabsf(v.w)))); }

// A block a row, a thread up to four float4 a block-width apart, kept in registers between the row's maximum and its planes.  scale[row]: what a product
// with the row is multiplied by.
// NORM: x = embedding row or x + partials (written back), planes of x * gain, scale with 1 / rms (run.cc:196-209).
// SWIGLU: silu(a) * c of the w1 | w3 partials (run.cc:344-347 order).  ROWS: src as it is.
enum { X3_NORM, X3_SWIGLU, X3_ROWS };
template <int MODE>
__global__ void __launch_bounds__(1024) x3_rows_kernel(X3RowsP p) {
  __shared__ float red[66];
  pdl_trigger();
  pdl_wait();
  const int b = blockIdx.x, n4 = p.n >> 2;
  const bool live = !p.pos || p.pos[b] >= 0;
  float4 v[4];
  float ss = 0.0f, m = 0.0f;
  if (MODE == X3_SWIGLU) {
    float4 c[4];
#pragma unroll
    for (int k = 0; k < 4; k++) {
      const int i = threadIdx.x + k * (int)blockDim.x;
      v[k] = c[k] = make_float4(0.f, 0.f, 0.f, 0.f);
      if (i < n4 && live)
        for (int z = 0; z < p.nz; z++) {
          const float* row = p.part + (size_t)z * p.zstride + (size_t)b * p.ld;
          const float4 az = ldg_stream(reinterpret_cast<const float4*>(row) + i), cz = ldg_stream(reinterpret_cast<const float4*>(row + p.n) + i);
          v[k].x += az.x; v[k].y += az.y; v[k].z += az.z; v[k].w += az.w;
          c[k].x += cz.x; c[k].y += cz.y; c[k].z += cz.z; c[k].w += cz.w;
        }
    }
#pragma unroll
    for (int k = 0; k < 4; k++) {
      v[k].x *= (1.0f / (1.0f + expf(-v[k].x))); v[k].x *= c[k].x;
      v[k].y *= (1.0f / (1.0f + expf(-v[k].y))); v[k].y *= c[k].y;
      v[k].z *= (1.0f / (1.0f + expf(-v[k].z))); v[k].z *= c[k].z;
      v[k].w *= (1.0f / (1.0f + expf(-v[k].w))); v[k].w *= c[k].w;
      m = x3_abs_max(v[k], m);
    }
  } else {
    float4* xr = reinterpret_cast<float4*>(p.x + (size_t)b * p.ld);
    const float4* src = MODE == X3_NORM && p.emb ? reinterpret_cast<const float4*>(p.emb + (size_t)p.token[b] * p.n) : xr;
#pragma unroll
    for (int k = 0; k < 4; k++) {
      const int i = threadIdx.x + k * (int)blockDim.x;
      v[k] = i < n4 && live ? src[i] : make_float4(0.f, 0.f, 0.f, 0.f);
    }
    if (MODE == X3_NORM) {
      for (int z = 0; z < p.nz && live; z++) {   // fixed order
        float4 pz[4];
#pragma unroll
        for (int k = 0; k < 4; k++) {
          const int i = threadIdx.x + k * (int)blockDim.x;
          pz[k] = i < n4 ? ldg_stream(reinterpret_cast<const float4*>(p.part + (size_t)z * p.zstride + (size_t)b * p.n) + i) : make_float4(0.f, 0.f, 0.f, 0.f);
        }
#pragma unroll
        for (int k = 0; k < 4; k++) { v[k].x += pz[k].x; v[k].y += pz[k].y; v[k].z += pz[k].z; v[k].w += pz[k].w; }
      }
    }
#pragma unroll
    for (int k = 0; k < 4; k++) {
      const int i = threadIdx.x + k * (int)blockDim.x;
      if (i >= n4) break;
      if (MODE == X3_NORM) {
        if (live && (p.emb || p.nz)) xr[i] = v[k];
        ss = dot4(v[k], v[k], ss);
        const float4 g = reinterpret_cast<const float4*>(p.gain)[i];
        v[k].x *= g.x; v[k].y *= g.y; v[k].z *= g.z; v[k].w *= g.w;
      }
      m = x3_abs_max(v[k], m);
    }
  }
  x3_block_sum_max(ss, m, red);
  float inverse;
  const float s = split_scale<X3_SCALE_MOST>(m, 14, &inverse);
#pragma unroll
  for (int k = 0; k < 4; k++) {
    const int i = threadIdx.x + k * (int)blockDim.x;
    if (i < n4) split_f16x4(v[k], s, reinterpret_cast<uint2*>(p.hi + (size_t)b * p.n)[i], reinterpret_cast<uint2*>(p.lo + (size_t)b * p.n)[i]);
  }
  if (threadIdx.x == 0) p.scale[b] = !live ? 0.0f : (MODE == X3_NORM ? inverse * (1.0f / sqrtf(ss / p.n + 1e-5f)) : inverse);
}

template <int MODE>
static int x3_rows_launch(cudaStream_t st, bool pdl, int rows, const X3RowsP& p) {
  int threads = ceil_div(p.n, 16 * 32) * 32;
  if (threads < 64) threads = 64;
  THA_CUDA_OK(launch(x3_rows_kernel<MODE>, dim3(rows), dim3(threads), 0, st, pdl, p));
  return THA_STATUS_SUCCESS;
}
int x3_norm_launch(cudaStream_t st, bool pdl, int rows, const X3RowsP& p) { return x3_rows_launch<X3_NORM>(st, pdl, rows, p); }
int x3_swiglu_launch(cudaStream_t st, bool pdl, int rows, const X3RowsP& p) { return x3_rows_launch<X3_SWIGLU>(st, pdl, rows, p); }
int x3_split_launch(cudaStream_t st, bool pdl, int rows, const X3RowsP& p) { return x3_rows_launch<X3_ROWS>(st, pdl, rows, p); }

// ---- host side ---------------------------------------------------------------------------------------------------------------
// Rows of planes start on 16 bytes (K a multiple of 8); a row fits the registers of a block of 1024 threads.
bool gemm_f16x3_width_ok(int K) { return K >= X3_BK && K % 8 == 0 && K <= 16 * 1024; }

static bool f16x3_ok(const X3Args& a) {
  if (a.n_mats < 1 || a.n_mats > 3 || a.N < 1 || !a.out || !a.colscale || !gemm_f16x3_width_ok(a.K)) return false;
  for (int i = 0; i < a.n_mats; i++)
    if (!a.W[i] || !aligned16(a.W[i]) || a.M[i] < 1) return false;
  return a.Xhi && a.Xlo && aligned16(a.Xhi) && aligned16(a.Xlo) && aligned16(a.colscale);
}

// Shares of K by the rounds that 74 pairs need, in k-blocks of a pair (0.43 us at most): an item costs its k-blocks and two more to start and to end; a share beyond the
// first costs its sums' way to memory and back (8 bytes a sum, at 6 TB/s).
int gemm_f16x3_splits(int tiles256, int rows_out, int K, int N) {
  const int kb = ceil_div(K, X3_BK), cells = tiles256 * ceil_div(N, X3_NT);
  int best = 1;
  float least = 0.0f;
  for (int z = 1; z <= 8 && kb / z >= 4; z++) {
    const int per = ceil_div(kb, z);
    if (ceil_div(kb, per) != z) continue;
    const float cost = (float)ceil_div(cells * z, 74) * ((float)per + 2.0f) + (float)(z - 1) * (float)rows_out * (float)N * 8.0f / 2.6e6f;
    if (z == 1 || cost < least) { least = cost; best = z; }
  }
  return best;
}

int gemm_f16x3_launch(cudaStream_t st, const X3Args& a, bool pdl) {
  if (!f16x3_ok(a)) return THA_STATUS_INVALID_ARG;
  CUtensorMap mw[3], mxh, mxl;
  X3P p = {};
  int tiles = 0;
  for (int i = 0; i < 3; i++) {
    if (i < a.n_mats) {
      THA_TRY_RC(tc_map(a.W[i], a.M[i], a.K, a.K, TC_BM, &mw[i]));
      p.W[i] = a.W[i]; p.M[i] = a.M[i]; p.tiles[i] = ceil_div(a.M[i], 2 * TC_BM); p.out_off[i] = a.out_off[i];
      tiles += p.tiles[i];
    } else {
      mw[i] = mw[0];
    }
  }
  THA_TRY_RC(tc_map(a.Xhi, a.N, a.K, a.K, X3_NT / 2, &mxh, 2));
  THA_TRY_RC(tc_map(a.Xlo, a.N, a.K, a.K, X3_NT / 2, &mxl, 2));
  p.K = a.K; p.N = a.N; p.ny = ceil_div(a.N, X3_NT);
  p.kblocks_total = ceil_div(a.K, X3_BK);
  p.splits = a.splits < 1 ? 1 : a.splits;
  p.kblocks_per_split = ceil_div(p.kblocks_total, p.splits);
  if (ceil_div(p.kblocks_total, p.kblocks_per_split) != p.splits) return THA_STATUS_INVALID_ARG;   // callers size their partial buffers by `splits`
  p.out = a.out; p.ldo = a.ldo; p.zstride = a.zstride; p.colscale = a.colscale;
  THA_TRY_RC(gemm_tc_init(&p.error_flag));
  p.n_items = tiles * p.ny * p.splits;
  const int pairs = p.n_items < 74 ? p.n_items : 74;
  THA_CUDA_OK(cudaFuncSetAttribute(gemm_f16x3_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, X3Smem::TOTAL));
  cudaLaunchConfig_t cfg = {};
  cudaLaunchAttribute attr[2];
  cfg.gridDim = dim3(2 * pairs); cfg.blockDim = dim3(X3_THREADS); cfg.dynamicSmemBytes = X3Smem::TOTAL; cfg.stream = st;
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = 2; attr[0].val.clusterDim.y = 1; attr[0].val.clusterDim.z = 1;
  attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[1].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr; cfg.numAttrs = pdl ? 2 : 1;
  count_launch();
  THA_CUDA_OK(cudaLaunchKernelEx(&cfg, gemm_f16x3_kernel, mw[0], mw[1], mw[2], mxh, mxl, p));
  trace_launch(reinterpret_cast<const void*>(gemm_f16x3_kernel), st);
  return THA_STATUS_SUCCESS;
}

}  // namespace tha

using namespace tha;

// C-ABI: out[z][n * ldo + row] = the z-th share of sum_k W[row, k] X[n, k]; hi, lo [N, K] and scale [N] are the caller's scratch
extern "C" int tha_gemm_f16x3(void* stream, float* out, long long ldo, const float* W, int M, int K, const float* X, int N, long long ldx, int splits,
                              uint16_t* hi, uint16_t* lo, float* scale) {
  if (!X || ldx < K || ldx % 4 || !aligned16(X) || !hi || !lo || !scale) return THA_STATUS_INVALID_ARG;
  X3Args a = {};
  a.n_mats = 1; a.W[0] = W; a.M[0] = M; a.K = K; a.Xhi = hi; a.Xlo = lo; a.N = N; a.colscale = scale; a.out = out; a.ldo = ldo;
  a.zstride = (long long)N * ldo; a.splits = splits;
  if (!f16x3_ok(a)) return THA_STATUS_INVALID_ARG;
  X3RowsP r = {};
  r.x = const_cast<float*>(X); r.ld = ldx; r.n = K; r.hi = hi; r.lo = lo; r.scale = scale;
  THA_TRY_RC(x3_split_launch((cudaStream_t)stream, false, N, r));
  return gemm_f16x3_launch((cudaStream_t)stream, a, false);
}
