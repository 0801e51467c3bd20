// Causal attention for batched prompt ingestion ON THE TENSOR CORES (bf16 model path): Q K^T and P V as
// tcgen05.mma.kind::f16 with fp32 accumulators in TMEM, softmax in fp32 registers between them.
//
// Rule (restated by the oracle, oracle/llama2_oracle.c orc_attention_bf16_tiled; reference arithmetic: run.cc:288-321):
// keys are visited in tiles of 128 starting at key 0; q, k, v are rounded to bf16 (nearest even); scores, the running
// maximum m, the running sum l and the output accumulator are fp32; per tile  p = exp(s - m_new)  is rounded to bf16 for
// the P V product, l accumulates the UNROUNDED p;  out = acc / l.
//
// q, K and V of the call's rows are left as bf16 rows by the kernel that rotates them (tc_rope_scatter_kernel), K and V of
// earlier positions by bf_kv_context_kernel (step_bf16.cu); every tile here is a TMA load of swizzled rows.  V is the B
// operand as it lies (key rows, channels contiguous: MN-major), P the A operand in TMEM, over the scores that it came from.
//
// CTA = 128 consecutive query rows of one (sequence, head), 256 threads, two CTAs an SM: two threads per query row (= TMEM
// lane), each with half of the row's key columns and half of its head-dimension accumulator.  A CTA is a chain -- S,
// maximum, weights, P V, accumulator -- in which only the loads of the next tile and its S (under the accumulator's update)
// run ahead; the other CTA of the SM fills it.  96 KB of shared memory (one K, one V buffer: each is free as soon as its
// product is done) and 256 TMEM columns each.
// Llama-2-7B layer, prompts of 777 and 2048 rows: 87 us; one CTA an SM with two K and two V^T buffers and P through shared
// memory took 250, and 58 more for a kernel that transposed V.  Eight portions of 16 rows behind contexts of 1000, where K and V were converted by
// every CTA: a step of two layers 705 -> 504 us.
#include <cuda.h>

#include "common.cuh"
#include "gemm_tc.h"
#include "tc_common.cuh"
#include "workspace.h"

namespace tha {

struct AttnPfTcP {
  uint16_t* out; int dim;                      // [rows, dim]: the row rounded to bf16 (wo's input)
  int kv_mul;
  const int* row_pos; const int* row_stage;    // [rows]: position; staged row of it
  const int* tile_row0; const int* tile_n;     // [tiles]: first row and row count (<= 128)
  int* error_flag;
};

constexpr int PTC_TQ = 128, PTC_TK = 128;

// two fp32 -> packed bf16x2, round to nearest even (one instruction; a in the low half)
__device__ __forceinline__ uint32_t ptc_bf16x2(float a, float b) {
  uint32_t r;
  asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(r) : "f"(b), "f"(a));
  return r;
}
__device__ __forceinline__ void ptc_tmem_ld32(uint32_t taddr, uint32_t (&v)[32]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16, %17, %18, %19, "
      "%20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
      : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]), "=r"(v[8]), "=r"(v[9]),
        "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15]), "=r"(v[16]), "=r"(v[17]), "=r"(v[18]), "=r"(v[19]),
        "=r"(v[20]), "=r"(v[21]), "=r"(v[22]), "=r"(v[23]), "=r"(v[24]), "=r"(v[25]), "=r"(v[26]), "=r"(v[27]), "=r"(v[28]), "=r"(v[29]),
        "=r"(v[30]), "=r"(v[31])
      : "r"(taddr));
}
// kind::f16, bf16 x bf16 -> fp32, both K-major, M = 128, N = n
__host__ __device__ constexpr uint32_t ptc_idesc(int n) {
  return (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(n >> 3) << 17) | ((uint32_t)(128 >> 4) << 24);
}
__device__ __forceinline__ void ptc_tmem_st16(uint32_t taddr, const uint32_t (&v)[16]) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16};"
      ::"r"(taddr), "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7]), "r"(v[8]), "r"(v[9]),
        "r"(v[10]), "r"(v[11]), "r"(v[12]), "r"(v[13]), "r"(v[14]), "r"(v[15]) : "memory");
}
// MN-major B, SWIZZLE_128B: blocks of 64 columns x 8 rows of K; K groups 1024 bytes apart, column blocks `block` bytes
__device__ __forceinline__ uint64_t ptc_desc_mn(uint32_t saddr, uint32_t block) {
  return (uint64_t)((saddr & 0x3FFFFu) >> 4) | (uint64_t)(block >> 4) << 16 | (uint64_t)(1024 >> 4) << 32 | (uint64_t)1 << 46 | (uint64_t)2 << 61;
}

template <int HS>
__global__ void __launch_bounds__(256, 2)
attn_prefill_tc_kernel(const __grid_constant__ CUtensorMap mq, const __grid_constant__ CUtensorMap mk, const __grid_constant__ CUtensorMap mv,
                       const AttnPfTcP p) {
  constexpr int KBH = HS / 64;                       // 64-value blocks along the head dimension
  constexpr int TILE = KBH * 128 * 128;              // Q, K and V tiles: [block][128 rows][128 bytes]
  constexpr int TMEM_COLS = 256;                     // S (and P over it): 128 columns, P V: HS columns
  constexpr int HH = HS / 2;                         // head-dimension columns per thread
  extern __shared__ unsigned char ptc_raw[];
  __shared__ float s_max[2][PTC_TQ];                 // row maxima / sums of the two column halves
  __shared__ uint64_t qbar, kbar, vbar, sbar, pbar;
  __shared__ uint32_t tmem_slot;
  __shared__ int abort_s, key_tiles;                 // key_tiles: of K, and of V, that are asked for; thread 0's
  unsigned char* smem = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(ptc_raw) + 1023) & ~(uintptr_t)1023);
  unsigned char *Qs = smem, *Ks = smem + TILE, *Vs = smem + 2 * TILE;

  // 8 warps: warp w serves TMEM lanes 32 (w & 3) .. (query rows) and column half w >> 2
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int qd = warp & 3, hf = warp >> 2;
  const int row = qd * 32 + lane;
  const int tile = (int)gridDim.y - 1 - (int)blockIdx.y, h = blockIdx.x;   // the last tiles of a prompt see the most keys: they start first
  if (tid == 0) {
    tc_mbar_init(&qbar, 1); tc_mbar_init(&kbar, 1); tc_mbar_init(&vbar, 1); tc_mbar_init(&sbar, 1); tc_mbar_init(&pbar, 1);
    abort_s = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    asm volatile("prefetch.tensormap [%0];" ::"l"(&mq) : "memory");
    asm volatile("prefetch.tensormap [%0];" ::"l"(&mk) : "memory");
    asm volatile("prefetch.tensormap [%0];" ::"l"(&mv) : "memory");
  }
  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(tc_smem_u32(&tmem_slot)), "r"(TMEM_COLS));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::);
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem_s = tmem_slot, tmem_pv = tmem_s + 128;
  int* abort_flag = &abort_s;
  pdl_wait();
  pdl_trigger();

  const int row0 = p.tile_row0[tile], n = p.tile_n[tile];
  const int pos0 = p.row_pos[row0];
  const bool live_tile = pos0 >= 0 && n > 0;
  const int kh = h / p.kv_mul;
  const int kmax = live_tile ? pos0 + n - 1 : -1;
  const int key_row0 = p.row_stage[row0] - pos0;     // staged row of position 0
  const float scale_log2 = 1.4426950408889634f / sqrtf((float)HS);   // scores in units of log2(e): exp(x) = exp2(x * log2 e)
  auto load = [&](unsigned char* dst, const CUtensorMap* m, int col, int r, uint64_t* bar) {
    tc_mbar_expect_tx(bar, TILE);
#pragma unroll
    for (int kb = 0; kb < KBH; kb++) tc_tma_2d(dst + kb * (128 * 128), m, col + kb * 64, r, bar);
  };
  auto scores = [&]() {
    constexpr uint32_t idesc = ptc_idesc(PTC_TK);
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
#pragma unroll
    for (int kb = 0; kb < KBH; kb++) {
      const uint64_t a = tc_smem_desc(tc_smem_u32(Qs + kb * (128 * 128))), b = tc_smem_desc(tc_smem_u32(Ks + kb * (128 * 128)));
#pragma unroll
      for (int k = 0; k < 4; k++) tc_mma_f16(tmem_s, a + (uint64_t)(2 * k), b + (uint64_t)(2 * k), idesc, (uint32_t)((kb | k) != 0));
    }
    tc_commit(&sbar);
  };
  if (tid == 0) key_tiles = live_tile ? kmax / PTC_TK + 1 : 0;
  bool ok = true;
  if (warp == 0 && live_tile) {
    if (tc_elect()) {
      load(Qs, &mq, h * HS, row0, &qbar);
      load(Ks, &mk, kh * HS, key_row0, &kbar);
      load(Vs, &mv, kh * HS, key_row0, &vbar);
      if (tc_mbar_wait(&qbar, 0u, abort_flag) && tc_mbar_wait(&kbar, 0u, abort_flag)) scores();
    }
    __syncwarp();
  }
  float m_run = -INFINITY, l_run = 0.0f;             // l_run: this thread's half of the row sum (both halves share m)
  float acc[HH];
#pragma unroll
  for (int c = 0; c < HH; c++) acc[c] = 0.0f;
  const int qpos = pos0 + (row < n ? row : n - 1);
  const uint32_t ts = tmem_s + ((uint32_t)(qd * 32) << 16) + (uint32_t)(64 * hf);
  const uint32_t tpv = tmem_pv + ((uint32_t)(qd * 32) << 16) + (uint32_t)(HH * hf);
  unsigned ph = 0;                                   // parity of this tile's phases
  for (int t0 = 0; t0 <= kmax; t0 += PTC_TK, ph ^= 1u) {
    const bool more = t0 + PTC_TK <= kmax, whole = t0 + PTC_TK - 1 <= pos0;   // whole: every row sees every key
    if (ok) ok = tc_mbar_wait(&sbar, ph, abort_flag);
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    if (warp == 0) {
      if (more && tc_elect()) load(Ks, &mk, kh * HS, key_row0 + t0 + PTC_TK, &kbar);
      __syncwarp();
    }
    // ---- softmax of this thread's half row (keys 64 hf .. 64 hf + 63 of the tile): the maximum first (exchanged with the
    // other half through shared memory), then, out of TMEM again, exponentials -> P (bf16) over the scores that they came from
    const int tk = t0 + 64 * hf;                     // first key of this thread's columns
    float mt = -INFINITY;
#pragma unroll
    for (int half = 0; half < 2; half++) {
      uint32_t s[32];
      ptc_tmem_ld32(ts + (uint32_t)(32 * half), s);
      asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
      if (whole) {
#pragma unroll
        for (int j = 0; j < 32; j++) mt = fmaxf(mt, __uint_as_float(s[j]) * scale_log2);
      } else {
#pragma unroll
        for (int j = 0; j < 32; j++)
          if (tk + 32 * half + j <= qpos) mt = fmaxf(mt, __uint_as_float(s[j]) * scale_log2);
      }
    }
    s_max[hf][row] = mt;
    __syncthreads();
    const float m_new = fmaxf(m_run, fmaxf(s_max[0][row], s_max[1][row]));   // finite: key 0 is visible to every row
    const float corr = exp2f(m_run - m_new);         // exp2(-inf) = 0 on the first tile
    float lsum = 0.0f;
#pragma unroll
    for (int half = 0; half < 2; half++) {
      uint32_t s[32], w[16];
      ptc_tmem_ld32(ts + (uint32_t)(32 * half), s);
      asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
      for (int j = 0; j < 32; j += 2) {
        float p0 = exp2f(__fsub_rn(__fmul_rn(__uint_as_float(s[j]), scale_log2), m_new));
        float p1 = exp2f(__fsub_rn(__fmul_rn(__uint_as_float(s[j + 1]), scale_log2), m_new));
        if (!whole) {
          if (tk + 32 * half + j > qpos) p0 = 0.0f;
          if (tk + 32 * half + j + 1 > qpos) p1 = 0.0f;
        }
        lsum += p0;
        lsum += p1;
        w[j >> 1] = ptc_bf16x2(p0, p1);
      }
      ptc_tmem_st16(ts + (uint32_t)(16 * half), w);
    }
    asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
    l_run = l_run * corr + lsum;
    m_run = m_new;
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    // ---- P V: keys 16 x .. 16 x + 15 of P are 8 columns, behind 64 hf for each half; groups of 16 behind the tile's last key are left out
    if (warp == 0) {
      if (tc_elect() && tc_mbar_wait(&vbar, ph, abort_flag)) {
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        constexpr uint32_t idesc = ptc_idesc(HS) | (1u << 16);
        const uint64_t b = ptc_desc_mn(tc_smem_u32(Vs), 128 * 128);
        const int groups = more ? PTC_TK / 16 : (kmax - t0 + 16) / 16;
        for (int x = 0; x < groups; x++)
          tc_mma_f16_ts(tmem_pv, tmem_s + (uint32_t)(64 * (x >> 2) + 8 * (x & 3)), b + (uint64_t)(x * (2048 >> 4)), idesc, (uint32_t)(x != 0));
        tc_commit(&pbar);
      }
      __syncwarp();
    }
    if (ok) ok = tc_mbar_wait(&pbar, ph, abort_flag);
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    if (warp == 0) {
      if (more && tc_elect()) {
        load(Vs, &mv, kh * HS, key_row0 + t0 + PTC_TK, &vbar);
        if (tc_mbar_wait(&kbar, ph ^ 1u, abort_flag)) scores();   // the next tile's, under this one's accumulator
      }
      __syncwarp();
    }
#pragma unroll
    for (int c0 = 0; c0 < HH; c0 += 32) {
      uint32_t v[32];
      ptc_tmem_ld32(tpv + (uint32_t)c0, v);
      asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
      for (int j = 0; j < 32; j++) acc[c0 + j] = acc[c0 + j] * corr + __uint_as_float(v[j]);
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  }

  // ---- the row sum is the sum of its two halves; normalise and store this thread's half row
  __syncthreads();
  s_max[hf][row] = l_run;
  __syncthreads();
  if (live_tile && row < n && ok) {
    const float inv = 1.0f / (s_max[0][row] + s_max[1][row]);
    uint16_t* orow = p.out + (size_t)(row0 + row) * p.dim + h * HS + HH * hf;
#pragma unroll
    for (int c = 0; c < HH; c += 8)
      *reinterpret_cast<uint4*>(orow + c) = make_uint4(ptc_bf16x2(acc[c] * inv, acc[c + 1] * inv), ptc_bf16x2(acc[c + 2] * inv, acc[c + 3] * inv),
                                                       ptc_bf16x2(acc[c + 4] * inv, acc[c + 5] * inv), ptc_bf16x2(acc[c + 6] * inv, acc[c + 7] * inv));
  }
  if (tid == 0 && *((volatile int*)&abort_s) && key_tiles) {
    tc_drain(&qbar, 1, 1);
    tc_drain(&kbar, 1, key_tiles);
    tc_drain(&vbar, 1, key_tiles);
  }
  __syncthreads();
  if (warp == 0) {
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_s), "r"(TMEM_COLS));
  }
  if (tid == 0 && abort_s && p.error_flag) *((volatile int*)p.error_flag) = 1;
}

bool attn_prefill_tc_supported(int head_size, int kv_dim) { return (head_size == 64 || head_size == 128) && kv_dim % 4 == 0; }

// tiles of up to 128 query rows (tile_row0 / tile_n), never across sequences; q16 [rows][dim], k16 / v16 [staged_rows][kv_dim]
// in bf16; row_stage: the staged row of every row (a sequence's staged rows begin at its position 0, at a multiple of 128)
int attn_prefill_tc_launch(cudaStream_t stream, int n_tiles, int rows, int n_heads, int n_kv_heads, int head_size, const uint16_t* q16,
                           uint16_t* out, const int* row_pos, const int* tile_row0, const int* tile_n, bool pdl, const uint16_t* k16,
                           const uint16_t* v16, int staged_rows, const int* row_stage) {
  if (!attn_prefill_tc_supported(head_size, n_kv_heads * head_size)) return THA_STATUS_NOT_SUPPORTED;
  AttnPfTcP p;
  p.out = out; p.dim = n_heads * head_size; p.kv_mul = n_heads / n_kv_heads;
  p.row_pos = row_pos; p.row_stage = row_stage; p.tile_row0 = tile_row0; p.tile_n = tile_n;
  THA_TRY_RC(gemm_tc_init(&p.error_flag));
  const int kvd = n_kv_heads * head_size;
  CUtensorMap mq, mk, mv;
  THA_TRY_RC(tc_map(q16, rows, p.dim, p.dim, 128, &mq, 2));
  THA_TRY_RC(tc_map(k16, staged_rows, kvd, kvd, 128, &mk, 2));
  THA_TRY_RC(tc_map(v16, staged_rows, kvd, kvd, 128, &mv, 2));
  const size_t smem = (size_t)3 * head_size * 256 + 1024;
  auto k = head_size == 64 ? attn_prefill_tc_kernel<64> : attn_prefill_tc_kernel<128>;
  THA_CUDA_OK(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  THA_CUDA_OK(launch(k, dim3(n_heads, n_tiles), dim3(256), smem, stream, pdl, mq, mk, mv, p));
  return THA_STATUS_SUCCESS;
}

}  // namespace tha
