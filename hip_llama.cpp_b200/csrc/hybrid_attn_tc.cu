// Softmax attention of prompt portions on the 5th-generation tensor cores (tcgen05 + TMEM) for the layer-program path: the bf16 number
// format, heads of 64 or 128 channels (keys and values alike).  The same numbers as hyb_attn_mma_kernel (hybrid_ops.cu), which keeps the short
// portions and the other head sizes: q, keys and values rounded to bf16, scores, softmax and sums in fp32, the weights either rounded to bf16
// or (EXACT) as two bf16 that carry 16 bits of them.
//
// A step's keys and values are rounded once, row by row, into scratch (hyb_attn_stage_kernel), from where tiles of 64 keys come by TMA.  A CTA
// takes 256 (position, query head) pairs of one key/value head: two groups of 128 rows that share every tile.  Ten warps:
//   0 .. 3, 4 .. 7  softmax of group 0 and 1, a thread a row: 64 scores out of TMEM, scale, bias, mask, weights back into the same TMEM columns as
//                   the A operand of the second product.  The accumulator stays in TMEM and is rescaled where a row's maximum grows.
//   8               one elected thread fetches tiles
//   9               one elected thread issues the products: scores of tile j + 1 ahead of weights x values of tile j, so that one group's softmax
//                   runs under the other's products
// TMEM: per group two score buffers of 64 columns and an accumulator of up to 128.  Values are the B operand as they lie (key rows, channels
// contiguous: MN-major), so nothing is transposed.  The distance biases of a block's heads stay in shared memory.
//
// Bound: the softmax, a chain of 2900 cycles a tile and group with two warps a scheduler; the products (EXACT: three of 128 x 64 x 128 a tile and
// group) take two thirds of that.  Prompts of 1100 and 2900, 16 heads of 128 on 4 with biases: 515 us a layer on mma.sync, 120 here.  (Cache rows
// fetched and rounded by warps of the CTA instead of staged: 205 to 450 us, the 28 KB that are left to L1 hold too few loads in flight.)
#include <cuda.h>

#include "gemm_tc.h"
#include "hybrid_ops.cuh"
#include "tc_common.cuh"

namespace tha {

constexpr int AT_KEYS = 64, AT_ROWS = 128, AT_STAGES = 3, AT_THREADS = 320;

__host__ __device__ constexpr int at_kv_stage(int DT) { return 2 * AT_KEYS * DT * 2; }
// a head's biases by distance, from -(AP + 31) to rel_n + AP + 31 (the ends repeated: no index is clamped), 8 banks from one head to the next
__host__ __device__ inline int at_rel_pad(int AP) { return AP + 32; }
__host__ __device__ inline int at_rel_pitch(int AP, int rel_n) { return (rel_n + 2 * at_rel_pad(AP) - 8 + 31) / 32 * 32 + 8; }
__host__ __device__ inline long long at_smem(int DT, int AG, int AP, int rel_n) {
  return 2ll * AT_ROWS * DT * 2 + AT_STAGES * at_kv_stage(DT) + (rel_n > 0 ? 4ll * AG * at_rel_pitch(AP, rel_n) : 0) + 1024;
}

__device__ __forceinline__ uint32_t at_bf16x2(float lo, float hi) {
  uint32_t r;
  asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(r) : "f"(hi), "f"(lo));
  return r;
}
__device__ __forceinline__ float at_ex2(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
// element (row r, column c) of a tile of 128-byte rows (64 bf16), SWIZZLE_128B
__device__ __forceinline__ int at_off(int r, int c) { return r * 128 + (((c >> 3) ^ (r & 7)) << 4) + ((c & 7) << 1); }
__device__ __forceinline__ void at_ld32(uint32_t taddr, uint32_t (&v)[32]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16, %17, %18, %19, "
      "%20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
      : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]), "=r"(v[8]), "=r"(v[9]),
        "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15]), "=r"(v[16]), "=r"(v[17]), "=r"(v[18]), "=r"(v[19]),
        "=r"(v[20]), "=r"(v[21]), "=r"(v[22]), "=r"(v[23]), "=r"(v[24]), "=r"(v[25]), "=r"(v[26]), "=r"(v[27]), "=r"(v[28]), "=r"(v[29]),
        "=r"(v[30]), "=r"(v[31])
      : "r"(taddr));
}
__device__ __forceinline__ void at_st16(uint32_t taddr, const uint32_t (&v)[16]) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16};"
      ::"r"(taddr), "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7]), "r"(v[8]), "r"(v[9]),
        "r"(v[10]), "r"(v[11]), "r"(v[12]), "r"(v[13]), "r"(v[14]), "r"(v[15]) : "memory");
}
__device__ __forceinline__ void at_wait_ld() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }
__device__ __forceinline__ void at_wait_st() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }
__device__ __forceinline__ void at_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void at_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
// kind::f16, bf16 x bf16 -> fp32, M = 128; b_mn: the B operand's N runs along its rows
__host__ __device__ constexpr uint32_t at_idesc(int n, int b_mn) {
  return (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)b_mn << 16) | ((uint32_t)(n >> 3) << 17) | ((uint32_t)(128 >> 4) << 24);
}
// MN-major B, SWIZZLE_128B: blocks of 64 columns (128 bytes) x 8 rows of K; K groups 1024 bytes apart, column blocks `block` bytes
__device__ __forceinline__ uint64_t at_desc_mn(uint32_t saddr, uint32_t block) {
  return (uint64_t)((saddr & 0x3FFFFu) >> 4) | (uint64_t)(block >> 4) << 16 | (uint64_t)(1024 >> 4) << 32 | (uint64_t)1 << 46 | (uint64_t)2 << 61;
}

// Where the staged rows of sequence `seq` begin: behind those of the sequences ahead of it that have min_rows rows in the step, each up to a multiple of 32.
__device__ __forceinline__ int at_stage_rows(const tha_rows_t& rows, int s, int min_rows) {
  const int lo = rows.seq_first[s], hi = rows.seq_first[s + 1];
  return hi - lo >= min_rows ? (rows.pos[hi - 1] + 32) / 32 * 32 : 0;
}
__device__ __forceinline__ int at_stage_base(const tha_rows_t& rows, int seq, int min_rows) {
  int sum = 0;
  for (int s = threadIdx.x & 31; s < seq; s += 32) sum += at_stage_rows(rows, s, min_rows);
  return __reduce_add_sync(THA_FULL_MASK, sum);
}

// Cache rows 0 .. p of every such sequence as bf16: k16, v16 [staged row][width]; a warp a row, zeros from the sequence's end to the next multiple of 32
// (weights of 0 meet them in the products).  grid (staged rows / 8)
__global__ void __launch_bounds__(256) hyb_attn_stage_kernel(tha_rows_t rows, tha_kv_t kv, int cache_layer, int kw, int vw, int min_rows, __nv_bfloat16* __restrict__ k16,
                                                             __nv_bfloat16* __restrict__ v16) {
  hyb_pdl_enter();
  const int lane = threadIdx.x & 31, row = blockIdx.x * 8 + (threadIdx.x >> 5);
  int seq = -1, t = row;
  for (int s0 = 0; s0 < rows.n_seqs && seq < 0; s0 += 32) {   // the sequence whose staged rows hold this one
    const int mine = s0 + lane < rows.n_seqs ? at_stage_rows(rows, s0 + lane, min_rows) : 0;
    int upto = mine;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) { const int v = __shfl_up_sync(THA_FULL_MASK, upto, o); if (lane >= o) upto += v; }
    const unsigned past = __ballot_sync(THA_FULL_MASK, upto > t);
    if (past) {
      const int i = __ffs(past) - 1;
      seq = s0 + i;
      t -= __shfl_sync(THA_FULL_MASK, upto - mine, i);
    } else {
      t -= __shfl_sync(THA_FULL_MASK, upto, 31);
    }
  }
  if (seq < 0) return;
  const int last = rows.pos[rows.seq_first[seq + 1] - 1];
  const size_t from = t <= last ? hyb_kv_row(kv, rows.seq_slot[seq], t, cache_layer) : (size_t)-1;
  auto copy = [&](const float* pool, int width, __nv_bfloat16* dst) {
    for (int c0 = 4 * lane; c0 < width; c0 += 512) {
      float4 v[4];
#pragma unroll
      for (int i = 0; i < 4; i++) {
        v[i] = make_float4(0.f, 0.f, 0.f, 0.f);
        if (c0 + 128 * i < width && from != (size_t)-1) v[i] = __ldg(reinterpret_cast<const float4*>(pool + from + c0 + 128 * i));
      }
#pragma unroll
      for (int i = 0; i < 4; i++)
        if (c0 + 128 * i < width)
          *reinterpret_cast<uint2*>(dst + (size_t)row * width + c0 + 128 * i) = make_uint2(at_bf16x2(v[i].x, v[i].y), at_bf16x2(v[i].z, v[i].w));
    }
  };
  copy(kv.k_pool, kw, k16);
  copy(kv.v_pool, vw, v16);
}

template <bool EXACT, bool CAP, bool REL, int DT>
__global__ void __launch_bounds__(AT_THREADS, 1) hyb_attn_tc_kernel(const __grid_constant__ CUtensorMap mk, const __grid_constant__ CUtensorMap mv, tha_attn_t a, tha_rows_t rows, const float* __restrict__ q,
                                                                    __nv_bfloat16* __restrict__ out, int AG, int AP, const float* __restrict__ gate,
                                                                    long long ldg, int min_rows, int* error_flag) {
  constexpr int KB = DT / 64;                        // 64-channel blocks
  constexpr int Q_GROUP = KB * AT_ROWS * 128, K_STAGE = AT_KEYS * DT * 2, KV_STAGE = 2 * K_STAGE;
  constexpr float LOG2E = 1.4426950408889634f;
  extern __shared__ unsigned char at_raw[];
  unsigned char* smem = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(at_raw) + 1023) & ~(uintptr_t)1023);
  unsigned char* Qs = smem;                          // [group][block][row][128 bytes]
  unsigned char* KVs = Qs + 2 * Q_GROUP;             // [stage][K | V][block][key][128 bytes]
  float* Bs = reinterpret_cast<float*>(KVs + AT_STAGES * KV_STAGE);   // biases [head][pitch]
  __shared__ uint64_t kv_full[AT_STAGES], kv_empty[AT_STAGES], s_full[2][2], p_full[2][2], pv_done[2][2];
  __shared__ uint32_t tmem_slot;
  __shared__ int abort_s;

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (threadIdx.x == 0) {
    for (int i = 0; i < AT_STAGES; i++) { tc_mbar_init(&kv_full[i], 1); tc_mbar_init(&kv_empty[i], 1); }
    for (int w = 0; w < 2; w++)
      for (int b = 0; b < 2; b++) { tc_mbar_init(&s_full[w][b], 1); tc_mbar_init(&p_full[w][b], 4); tc_mbar_init(&pv_done[w][b], 1); }
    abort_s = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  }
  // All of the SM's TMEM, ahead of the trigger: the product behind this kernel may start on this SM once every block has triggered, allocates its own columns
  // at once and keeps them until this grid has completed.  A block that came to its allocation after that would wait for ever (with heads of
  // 64 both fit an SM).
  if (warp == 9) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(tc_smem_u32(&tmem_slot)), "r"(512));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::);
  }
  at_fence_before();
  __syncthreads();
  at_fence_after();
  const uint32_t tmem = tmem_slot;
  hyb_pdl_enter();
  auto release = [&]() {
    if (warp == 9) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512));
  };
  int seq = -1, r0 = 0, r_end = 0;
  {
    // the last tiles of a prompt see the most keys: tile numbers in descending order over all sequences, so that the grid ends on short ones
    int i = (int)blockIdx.y, tile = 0;
    auto tiles_of = [&](int s) {
      const int n = rows.seq_first[s + 1] - rows.seq_first[s];
      return n >= min_rows ? (n + AP - 1) / AP : 0;
    };
    if (rows.n_seqs <= 32) {
      const int mine = lane < rows.n_seqs ? tiles_of(lane) : 0;
      for (int level = __reduce_max_sync(THA_FULL_MASK, mine) - 1; level >= 0; level--) {
        const unsigned has = __ballot_sync(THA_FULL_MASK, mine > level);
        if (i < __popc(has)) { seq = __fns(has, 0, i + 1); tile = level; break; }
        i -= __popc(has);
      }
    } else {
      for (int s = 0; s < rows.n_seqs; s++) {
        const int nt = tiles_of(s);
        if (i < nt) { seq = s; tile = nt - 1 - i; break; }
        i -= nt;
      }
    }
    if (seq < 0) { release(); return; }   // the same for the whole block
    r0 = rows.seq_first[seq] + tile * AP;
    r_end = min(rows.seq_first[seq + 1], r0 + AP);
  }
  const int g = blockIdx.x, gsize = a.heads / a.kv_heads;
  const int gv = a.v_share > 1 ? g / a.v_share : g;
  const int key_row0 = at_stage_base(rows, seq, min_rows);   // staged row of position 0
  const int p_first = rows.pos[r0], p_last = p_first + (r_end - r0) - 1;
  const int key_lo = a.chunk > 0 ? (p_first / a.chunk) * a.chunk : 0;
  const int last_first = a.chunk > 0 ? (p_last / a.chunk) * a.chunk : 0;
  const HybTiles tiles = hyb_attn_tiles(a, key_lo, p_first, p_last);   // of 32 keys: two to a tile here
  const int n = (tiles.n + 1) >> 1;
  auto half_key = [&](int ti) { return ti < tiles.n_a ? tiles.begin + 32 * ti : tiles.resume + 32 * (ti - tiles.n_a); };
  const int BP = REL ? at_rel_pitch(AP, a.rel_n) : 0, pad = at_rel_pad(AP);

  // q, rounded: warp w takes rows w, w + 10, ..; pairs past the block's positions are zeros
  for (int pr = warp; pr < 2 * AT_ROWS; pr += AT_THREADS / 32) {
    const int pp = pr / AG, hg = pr - pp * AG;
    const bool ok = pp < AP && r0 + pp < r_end;
    if (4 * lane < DT) {
      float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
      if (ok) v = *reinterpret_cast<const float4*>(q + ((size_t)(r0 + pp) * a.heads + (size_t)g * gsize + hg) * DT + 4 * lane);
      const int c = 4 * lane;
      *reinterpret_cast<uint2*>(Qs + (pr / AT_ROWS) * Q_GROUP + (c >> 6) * (AT_ROWS * 128) + at_off(pr % AT_ROWS, c & 63)) =
          make_uint2(at_bf16x2(v.x, v.y), at_bf16x2(v.z, v.w));
    }
  }
  if (REL) {
    const int count = min(a.rel_n, p_last + 1) + 2 * pad;   // distances past the block's farthest key are not asked for
    for (int hl = 0; hl < AG; hl++)
      for (int i = threadIdx.x; i < count; i += AT_THREADS) Bs[hl * BP + i] = hyb_attn_rel(a, g * gsize + hl, i - pad);
  }
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  __syncthreads();
  int* abort_flag = &abort_s;

  if (warp < 8) {
    // ===== softmax of group w
    const int w = warp >> 2, row = (warp & 3) * 32 + lane, pr = w * AT_ROWS + row;
    const int pp = pr / AG, hg = pr - pp * AG, h = g * gsize + hg;
    const bool row_ok = pp < AP && r0 + pp < r_end;
    const int pos = p_first + pp, first = a.chunk > 0 ? (pos / a.chunk) * a.chunk : 0;
    const float scale = a.scale * ((a.head_scale && row_ok) ? a.head_scale[h] : 1.0f);
    const float two_over_cap = CAP ? 2.0f / a.softcap : 0.f;
    const float far = REL && row_ok ? hyb_attn_rel(a, h, a.rel_n - 1) : 0.f;
    const uint32_t lanes = (uint32_t)((warp & 3) * 32) << 16;
    const uint32_t t_s = tmem + lanes + (uint32_t)(w * 2 * AT_KEYS), t_o = tmem + lanes + (uint32_t)(4 * AT_KEYS + w * DT);
    float m = -INFINITY, l = 0.f, shift = 0.f;       // weights: 2^(score log2(e) + shift), shift = -m log2(e) rounded; 0 while nothing was seen
    bool ok = true;
    for (int j = 0; j < n && ok; j++) {
      const int b = j & 1;
      ok = tc_mbar_wait(&s_full[w][b], (unsigned)(j >> 1) & 1u, abort_flag);
      ok = __all_sync(THA_FULL_MASK, ok);
      at_fence_after();
      float t[AT_KEYS];
      float mx = -INFINITY;
#pragma unroll
      for (int hf = 0; hf < 2; hf++) {
        uint32_t s[32];
        at_ld32(t_s + (uint32_t)(b * AT_KEYS + 32 * hf), s);
        const int ti = 2 * j + hf;
        const bool there = ti < tiles.n;
        const int kt = half_key(there ? ti : tiles.n - 1);   // behind the last half its own keys again, as fetched: the biases end there
        // every position of the block sees every key of this half
        const bool whole = there && kt + 31 <= p_first && kt >= last_first && (a.window <= 0 || p_last - kt < a.window || kt + 32 <= a.keep_first);
        const bool near = REL && p_first - (kt + 31) < a.rel_n - 1;   // the same for the whole block
        const float* bias = REL ? Bs + hg * BP + pad + (p_first + min(pp, AP - 1) - kt) : nullptr;
        at_wait_ld();
#pragma unroll
        for (int i = 0; i < 32; i++) {
          const float sv = __uint_as_float(s[i]);
          float x;
          if (CAP) x = a.softcap - __fdividef(2.0f * a.softcap, 1.0f + __expf(sv * scale * two_over_cap));
          else if (REL) x = fmaf(sv, scale, near ? bias[-i] : far);
          else x = sv * scale;
          t[32 * hf + i] = x;
        }
        if (!whole) {
#pragma unroll
          for (int i = 0; i < 32; i++)
            if (!(row_ok && there && hyb_attn_sees(a, kt + i, pos, first))) t[32 * hf + i] = -INFINITY;
        }
#pragma unroll
        for (int i = 0; i < 32; i++) mx = fmaxf(mx, t[32 * hf + i]);
      }
      const bool grow = mx > m;                       // also from -inf, where nothing was seen before
      if (__any_sync(THA_FULL_MASK, grow)) {
        const float to = grow ? -mx * LOG2E : shift;
        const float corr = m > -INFINITY ? at_ex2(to - shift) : grow ? 0.f : 1.f;
        m = grow ? mx : m;
        shift = to;
        l *= corr;
        if (j > 0) {   // all products of earlier tiles are in the accumulator
          ok = __all_sync(THA_FULL_MASK, tc_mbar_wait(&pv_done[w][b ^ 1], (unsigned)((j - 1) >> 1) & 1u, abort_flag) && ok);
          at_fence_after();
#pragma unroll
          for (int c = 0; c < DT; c += 32) {
            uint32_t o[32];
            at_ld32(t_o + (uint32_t)c, o);
            at_wait_ld();
#pragma unroll
            for (int i = 0; i < 32; i++) o[i] = __float_as_uint(__uint_as_float(o[i]) * corr);
            tc_tmem_st32(t_o + (uint32_t)c, o);
          }
        }
      }
      float sum = 0.f;
#pragma unroll
      for (int c = 0; c < AT_KEYS / 2; c += 16) {
        uint32_t hi[16], lo[16];
#pragma unroll
        for (int i = 0; i < 16; i++) {
          const float p0 = at_ex2(fmaf(t[2 * (c + i)], LOG2E, shift)), p1 = at_ex2(fmaf(t[2 * (c + i) + 1], LOG2E, shift));
          hi[i] = at_bf16x2(p0, p1);
          const float h0 = __uint_as_float(hi[i] << 16), h1 = __uint_as_float(hi[i] & 0xFFFF0000u);
          if (EXACT) {   // hi + lo carry 16 mantissa bits of the fp32 weight; the sum adds the fp32 weights themselves
            lo[i] = at_bf16x2(p0 - h0, p1 - h1);
            sum += p0 + p1;
          } else {
            sum += h0 + h1;
          }
        }
        at_st16(t_s + (uint32_t)(b * AT_KEYS + c), hi);
        if (EXACT) at_st16(t_s + (uint32_t)(b * AT_KEYS + 32 + c), lo);
      }
      l += sum;
      at_wait_st();
      at_fence_before();
      __syncwarp();
      if (lane == 0) tc_mbar_arrive(&p_full[w][b]);
    }
    if (ok) ok = tc_mbar_wait(&pv_done[w][(n - 1) & 1], (unsigned)((n - 1) >> 1) & 1u, abort_flag);
    at_fence_after();
    ok = __all_sync(THA_FULL_MASK, ok);
    float inv = 0.f;
    if (row_ok) {
      // all weights and their sum carry the factor 2^(m log2(e) + shift) of the rounded shift; the sink is weighed by m itself
      const float f = m > -INFINITY ? at_ex2(-fmaf(m, LOG2E, shift)) : 1.f;
      inv = f * hyb_attn_final_factor(a, h, m, l * f, gate ? gate + (size_t)(r0 + pp) * ldg : nullptr);
    }
#pragma unroll
    for (int c = 0; c < DT; c += 32) {
      uint32_t o[32];
      at_ld32(t_o + (uint32_t)c, o);
      at_wait_ld();
      if (row_ok && ok) {
        const size_t at = ((size_t)(r0 + pp) * a.heads + h) * DT + c;
        if (a.out_f32) {
          float* dst = reinterpret_cast<float*>(out) + at;
#pragma unroll
          for (int i = 0; i < 32; i += 4)
            *reinterpret_cast<float4*>(dst + i) = make_float4(__uint_as_float(o[i]) * inv, __uint_as_float(o[i + 1]) * inv, __uint_as_float(o[i + 2]) * inv,
                                                              __uint_as_float(o[i + 3]) * inv);
        } else {
          __nv_bfloat16* dst = out + at;
#pragma unroll
          for (int i = 0; i < 32; i += 8)
            *reinterpret_cast<uint4*>(dst + i) = make_uint4(at_bf16x2(__uint_as_float(o[i]) * inv, __uint_as_float(o[i + 1]) * inv),
                                                            at_bf16x2(__uint_as_float(o[i + 2]) * inv, __uint_as_float(o[i + 3]) * inv),
                                                            at_bf16x2(__uint_as_float(o[i + 4]) * inv, __uint_as_float(o[i + 5]) * inv),
                                                            at_bf16x2(__uint_as_float(o[i + 6]) * inv, __uint_as_float(o[i + 7]) * inv));
        }
      }
    }
    at_fence_before();
  } else if (warp == 8) {
    // ===== tiles: two halves of 32 keys, each a box of 64 channels at a time
    if (tc_elect()) {
      bool ok = true;
      for (int j = 0; j < n && ok; j++) {
        const int st = j % AT_STAGES;
        if (j >= AT_STAGES && !tc_mbar_wait(&kv_empty[st], (unsigned)(j / AT_STAGES - 1) & 1u, abort_flag)) { ok = false; tc_drain(kv_full, AT_STAGES, j); break; }
        tc_mbar_expect_tx(&kv_full[st], KV_STAGE);
#pragma unroll
        for (int hf = 0; hf < 2; hf++) {
          // behind the last half its own rows again: finite, and masked
          const int ti = 2 * j + hf < tiles.n ? 2 * j + hf : tiles.n - 1, key = key_row0 + half_key(ti);
          unsigned char* d = KVs + st * KV_STAGE + hf * 32 * 128;
#pragma unroll
          for (int kb = 0; kb < KB; kb++) {
            tc_tma_2d(d + kb * (AT_KEYS * 128), &mk, g * DT + kb * 64, key, &kv_full[st]);
            tc_tma_2d(d + K_STAGE + kb * (AT_KEYS * 128), &mv, gv * DT + kb * 64, key, &kv_full[st]);
          }
        }
      }
    }
  } else if (tc_elect()) {
    // ===== products
    constexpr uint32_t id_s = at_idesc(AT_KEYS, 0), id_o = at_idesc(DT, 1);
    const uint32_t q_addr = tc_smem_u32(Qs), kv_addr = tc_smem_u32(KVs);
    bool ok = true;
    auto scores = [&](int j, int w) {
      const uint32_t d = tmem + (uint32_t)(w * 2 * AT_KEYS + (j & 1) * AT_KEYS), k = kv_addr + (uint32_t)((j % AT_STAGES) * KV_STAGE);
#pragma unroll
      for (int kb = 0; kb < KB; kb++) {
        const uint64_t ad = tc_smem_desc(q_addr + (uint32_t)(w * Q_GROUP + kb * AT_ROWS * 128)), bd = tc_smem_desc(k + (uint32_t)(kb * AT_KEYS * 128));
#pragma unroll
        for (int x = 0; x < 4; x++) tc_mma_f16(d, ad + (uint64_t)(2 * x), bd + (uint64_t)(2 * x), id_s, (uint32_t)((kb | x) != 0));
      }
      tc_commit(&s_full[w][j & 1]);
    };
    ok = tc_mbar_wait(&kv_full[0], 0u, abort_flag);
    at_fence_after();
    if (ok) { scores(0, 0); scores(0, 1); }
    for (int j = 0; j < n && ok; j++) {
      if (j + 1 < n) {
        ok = tc_mbar_wait(&kv_full[(j + 1) % AT_STAGES], (unsigned)((j + 1) / AT_STAGES) & 1u, abort_flag);
        for (int w = 0; w < 2 && ok; w++) {
          if (j > 0) ok = tc_mbar_wait(&pv_done[w][(j + 1) & 1], (unsigned)((j - 1) >> 1) & 1u, abort_flag);   // the buffer's weights have been used
          at_fence_after();
          if (ok) scores(j + 1, w);
        }
      }
      for (int w = 0; w < 2 && ok; w++) {
        ok = tc_mbar_wait(&p_full[w][j & 1], (unsigned)(j >> 1) & 1u, abort_flag);
        at_fence_after();
        if (!ok) break;
        const uint32_t d = tmem + (uint32_t)(4 * AT_KEYS + w * DT), p = tmem + (uint32_t)(w * 2 * AT_KEYS + (j & 1) * AT_KEYS);
        const uint64_t vd = at_desc_mn(kv_addr + (uint32_t)((j % AT_STAGES) * KV_STAGE + K_STAGE), AT_KEYS * 128);
#pragma unroll
        for (int x = 0; x < AT_KEYS / 16; x++) {
          tc_mma_f16_ts(d, p + (uint32_t)(8 * x), vd + (uint64_t)(x * (2048 >> 4)), id_o, (uint32_t)((j | x) != 0));
          if (EXACT) tc_mma_f16_ts(d, p + (uint32_t)(32 + 8 * x), vd + (uint64_t)(x * (2048 >> 4)), id_o, 1u);
        }
        tc_commit(&pv_done[w][j & 1]);
      }
      tc_commit(&kv_empty[j % AT_STAGES]);
    }
  }
  __syncwarp();
  __syncthreads();
  at_fence_after();
  release();
  if (threadIdx.x == 0 && abort_s && error_flag) *((volatile int*)error_flag) = 1;
}

// Floats of scratch for the staged rows of a step (K and V rows of up to n_seqs contexts), 0: this form does not take the step.  A block's tiles come one
// after the other (1.6 us each, and 12 before the first), so there have to be enough of them: us with this form / hyb_attn_mma_kernel, heads of 128, 16 heads
// on 4: 128 rows 20 / 21, 256 rows 23 / 27, 1024 rows 43 / 112, 4096 rows 132 / 604; 8 heads on 2: 384 rows 26 / 24, 512 rows 29 / 37, 4096 rows
// 123 / 389; 16 heads of 64 on 16 (256 positions a block): 256 rows 35 / 20, 512 rows 41 / 44, 768 rows 47 / 63, 4096 rows 152 / 608; with biases, 16 on 4,
// 1024 rows 50 / 117; softcap and a window of 1024, 8 on 2, 2048 rows 70 / 141.  And no more cached rows to round than a few times the step's own.
size_t hyb_attn_tc_scratch(const tha_attn_t* a, const tha_rows_t* rows) {
  const int gsize = a->heads / a->kv_heads;
  if (a->dim != a->vdim || (a->dim != 64 && a->dim != 128) || gsize > 2 * AT_ROWS) return 0;
  const int AP = 2 * AT_ROWS / gsize;
  if ((long long)(rows->n_rows / AP) * a->kv_heads < (AP <= 85 ? 16 : 3 * AP / 16)) return 0;
  if (at_smem(a->dim, gsize, AP, a->rel ? a->rel_n : 0) > TC_SMEM_LIMIT - 1024) return 0;
  if (rows->n_rows / AP + rows->n_seqs > 65535) return 0;   // position tiles are the grid's second dimension
  const long long staged = (long long)rows->n_seqs * ((rows->max_pos + 32) / 32 * 32);
  if (staged > 4ll * rows->n_rows + 4096) return 0;
  return (size_t)staged * a->kv_heads * a->dim + 64;
}

template <bool EXACT, bool CAP, bool REL, int DT>
static int at_launch(cudaStream_t s, const tha_attn_t* a, const tha_rows_t* rows, const CUtensorMap& mk, const CUtensorMap& mv, const float* q, __nv_bfloat16* out,
                     const float* gate, long long ldg, int min_rows) {
  const int gsize = a->heads / a->kv_heads, AG = gsize, AP = 2 * AT_ROWS / AG;
  int* flag = nullptr;
  THA_TRY_RC(gemm_tc_init(&flag));
  const size_t smem = (size_t)at_smem(DT, AG, AP, REL ? a->rel_n : 0);
  auto k = hyb_attn_tc_kernel<EXACT, CAP, REL, DT>;
  THA_CUDA_OK(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  THA_CUDA_OK(launch(k, dim3(a->kv_heads, rows->n_rows / AP + rows->n_seqs), dim3(AT_THREADS), smem, s, pdl_enabled() != 0, mk, mv, *a, *rows, q, out, AG, AP, gate, ldg,
                     min_rows, flag));
  return THA_STATUS_SUCCESS;
}
template <int DT>
static int at_form(cudaStream_t s, const tha_attn_t* a, const tha_rows_t* rows, const CUtensorMap& mk, const CUtensorMap& mv, const float* q, __nv_bfloat16* out,
                   const float* gate, long long ldg, int min_rows) {
  if (a->rel) return at_launch<true, false, true, DT>(s, a, rows, mk, mv, q, out, gate, ldg, min_rows);
  if (a->softcap > 0.f) return at_launch<true, true, false, DT>(s, a, rows, mk, mv, q, out, gate, ldg, min_rows);
  if (a->fp32_scores) return at_launch<true, false, false, DT>(s, a, rows, mk, mv, q, out, gate, ldg, min_rows);
  return at_launch<false, false, false, DT>(s, a, rows, mk, mv, q, out, gate, ldg, min_rows);
}

// THA_STATUS_NOT_SUPPORTED (nothing launched): the caller takes another form.
int hyb_attn_tc_launch(cudaStream_t s, const tha_attn_t* a, const tha_rows_t* rows, const tha_kv_t* kv, const float* q, __nv_bfloat16* out, const float* gate,
                       long long ldg, int min_rows, float* scratch, size_t scratch_floats) {
  const size_t need = hyb_attn_tc_scratch(a, rows);
  if (!need || !scratch || scratch_floats < need || kv->kv_dim % 4 || !aligned16(kv->k_pool) || !aligned16(kv->v_pool) || !aligned16(q) || !aligned16(out))
    return THA_STATUS_NOT_SUPPORTED;   // 128-bit loads and stores
  const int staged = rows->n_seqs * ((rows->max_pos + 32) / 32 * 32);
  const int kw = a->kv_heads * a->dim, vw = a->kv_heads / (a->v_share > 1 ? a->v_share : 1) * a->dim;
  __nv_bfloat16* k16 = reinterpret_cast<__nv_bfloat16*>((reinterpret_cast<uintptr_t>(scratch) + 127) & ~(uintptr_t)127);
  __nv_bfloat16* v16 = k16 + (size_t)staged * kw;
  CUtensorMap mk, mv;
  THA_TRY_RC(tc_map(k16, staged, kw, kw, 32, &mk, 2));
  THA_TRY_RC(tc_map(v16, staged, vw, vw, 32, &mv, 2));
  THA_CUDA_OK(launch(hyb_attn_stage_kernel, dim3(staged / 8), dim3(256), 0, s, pdl_enabled() != 0, *rows, *kv, a->cache_layer, kw, vw, min_rows, k16, v16));
  return a->dim == 64 ? at_form<64>(s, a, rows, mk, mv, q, out, gate, ldg, min_rows) : at_form<128>(s, a, rows, mk, mv, q, out, gate, ldg, min_rows);
}

}  // namespace tha
