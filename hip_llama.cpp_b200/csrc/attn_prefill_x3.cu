// Causal attention of fp32 prompts on the tensor cores: Q K^T and P V as three fp16 products each of operands split in two (split_f16.cuh), softmax in fp32 between them, one pass over the keys as in attn_prefill.cu.
//
// x3_rope_kernel, which rotates q and k and fills the cache, leaves q, k and v of the call's rows as two fp16 planes besides, each (row, head) brought
// to [2^14, 2^15) by a power of two of its own; x3_context_kernel those of earlier positions.  A score is the product times the two inverse scales.  V's belong to
// the keys, so they go into the weights: a weight p becomes p vs / c, c the largest inverse scale of the tile's keys that the row sees, before it is split, and the row's P V
// of the tile is multiplied by c where it joins the accumulator in registers.  The corrections (hi.lo, lo.hi) of a product are summed ahead of hi.hi, which takes their sum
// over times 2^-11 (the MMA's scale of its input D).
//
// CTA = 128 consecutive query rows of one (sequence, head), 256 threads, two a row (attn_prefill_tc.cu); tiles of 128 keys.  A chain
// of S, softmax, P V and accumulator, in which the next tile's loads and its S run ahead; heads of 64 have two CTAs an SM (96 KB), of 128 one (192 KB).  Bound by that
// chain: issue slots 29 and 32 % busy, the tensor pipe 23 and 10 % (heads of 128, one prompt of 1024; of 64, 16 of 9 .. 201).  A layer of these 333 -> 61 us and 38 -> 21
// against attn_prefill.cu.
#include <cuda.h>

#include "common.cuh"
#include "gemm_tc.h"
#include "split_f16.cuh"
#include "tc_common.cuh"
#include "workspace.h"

namespace tha {

constexpr int AX_T = 128;                            // query rows and keys of a tile

struct AttnX3P {
  float* out; int dim, kv_mul, heads, staged_rows;
  const float *qs, *ks, *vs;                         // inverse scales: [rows][heads], [kv head][staged row]
  const int* row_pos; const int* row_stage;          // [rows]: position; staged row of it
  const int* tile_row0; const int* tile_n;           // [tiles]: first row and row count (<= 128)
  int* error_flag;
};

// The power of two that brings |v| to [2^14, 2^15) and its inverse.  At most 2^100: the ratio of two inverse scales stays finite.
__device__ __forceinline__ float ax_scale(float v, float* inverse) { return split_scale<100>(v, 14, inverse); }
__device__ __forceinline__ void ax_planes(float4 v, float s, uint16_t* hi, uint16_t* lo) {
  split_f16x4(v, s, *reinterpret_cast<uint2*>(hi), *reinterpret_cast<uint2*>(lo));
}
// Largest |value| of the head that this lane's four values belong to: hs / 4 neighbouring lanes
__device__ __forceinline__ float ax_head_max(float4 v, int hs) {
  float m = fmaxf(fmaxf(fabsf(v.x), fabsf(v.y)), fmaxf(fabsf(v.z), fabsf(v.w)));
  for (int o = hs >> 3; o > 0; o >>= 1) m = fmaxf(m, __shfl_xor_sync(THA_FULL_MASK, m, o));
  return m;
}

// tc_rope_scatter_kernel (step_tc.cu) for this attention: the same cache rows, to the bit, and the planes.  hs 64 or 128.
// Bound by memory as that one is; 16 bytes a value of q|k|v with one share of K.  grid (ld / 2048, rows)
__global__ void __launch_bounds__(256) x3_rope_kernel(const float* part, int nz, long long zstride, int ld, const int* pos, int d, int kvd, int hs,
                                                      const float* rc, const float* rs, float* kc, float* vc,
                                                      long long kv_bs, int loff, const int* slot, const KvPaged pg, const X3Staged st) {
  pdl_trigger();
  pdl_wait();
  const int b = blockIdx.y, pb = pos[b], sb = slot[b], staged = st.row[b];
  float4 v[2];
  int idx[2];
#pragma unroll
  for (int u = 0; u < 2; u++) {
    idx[u] = 4 * ((blockIdx.x * 2 + u) * blockDim.x + threadIdx.x);
    v[u] = make_float4(0.f, 0.f, 0.f, 0.f);
    if (idx[u] < d + 2 * kvd) {
#pragma unroll 4
      for (int z = 0; z < nz; z++) {
        const float4 pz = *reinterpret_cast<const float4*>(part + (size_t)z * zstride + (size_t)b * ld + idx[u]);
        v[u].x += pz.x; v[u].y += pz.y; v[u].z += pz.z; v[u].w += pz.w;
      }
    }
  }
  if (pb < 0) return;
  const long long rowoff = pg.table ? kv_paged_off(pg, sb, pb, kvd) : (long long)sb * kv_bs + loff + (long long)pb * kvd;
#pragma unroll
  for (int u = 0; u < 2; u++) {
    const int i = idx[u], part_of = i < d ? 0 : (i < d + kvd ? 1 : 2);       // of q, k, v
    const int li = part_of == 0 ? i : i - d - (part_of == 2 ? kvd : 0), head = li / hs;
    float4 r = v[u];
    if (part_of < 2) {
      const int j = (li % hs) >> 1;
      const float2 c = *reinterpret_cast<const float2*>(rc + (size_t)pb * (hs >> 1) + j), s = *reinterpret_cast<const float2*>(rs + (size_t)pb * (hs >> 1) + j);
      r = make_float4(fmaf(v[u].x, c.x, -__fmul_rn(v[u].y, s.x)), fmaf(v[u].x, s.x, __fmul_rn(v[u].y, c.x)),
                      fmaf(v[u].z, c.y, -__fmul_rn(v[u].w, s.y)), fmaf(v[u].z, s.y, __fmul_rn(v[u].w, c.y)));
    }
    float inverse;
    const float s = ax_scale(ax_head_max(r, hs), &inverse);
    if (i >= d + 2 * kvd) continue;
    const bool first = li % hs == 0;
    if (part_of == 0) {
      ax_planes(r, s, st.qh + (size_t)b * d + li, st.ql + (size_t)b * d + li);
      if (first) st.qs[(size_t)b * (d / hs) + head] = inverse;
      continue;
    }
    *reinterpret_cast<float4*>((part_of == 1 ? kc : vc) + rowoff + li) = r;
    const size_t at = (size_t)staged * kvd + li;
    ax_planes(r, s, (part_of == 1 ? st.kh : st.vh) + at, (part_of == 1 ? st.kl : st.vl) + at);
    if (first) (part_of == 1 ? st.ks : st.vs)[(size_t)head * st.rows + staged] = inverse;
    // behind a sequence's last row zeros to the end of its group of 16 keys: weights of 0 meet them there
    if (part_of == 2)
      for (int z = 1; z <= st.pad[b]; z++) {
        *reinterpret_cast<uint2*>(st.vh + at + (size_t)z * kvd) = make_uint2(0u, 0u);
        *reinterpret_cast<uint2*>(st.vl + at + (size_t)z * kvd) = make_uint2(0u, 0u);
      }
  }
}

// Cache rows of positions 0 .. upto[i] - 1 of sequence i -> planes and scales of staged rows base[i] + t.  grid (kvd / 1024, positions, sequences)
__global__ void __launch_bounds__(256) x3_context_kernel(const float* kc, const float* vc, long long kv_bs, const int* seq_slot,
                                                         const int* upto, const int* base, const KvPaged pg, int kvd, int hs, const X3Staged st) {
  pdl_trigger();
  pdl_wait();                                        // the call's own rows are in the cache
  const int i = blockIdx.z, n = upto[i], slot = seq_slot[i], li = 4 * (blockIdx.x * blockDim.x + threadIdx.x);
  for (int t = blockIdx.y; t < n; t += gridDim.y) {
    const long long off = pg.table ? kv_paged_off(pg, slot, t, kvd) : (long long)slot * kv_bs + (long long)t * kvd;
    float4 k = make_float4(0.f, 0.f, 0.f, 0.f), v = k;
    if (li < kvd) {
      k = *reinterpret_cast<const float4*>(kc + off + li);
      v = *reinterpret_cast<const float4*>(vc + off + li);
    }
    float ik, iv;
    const float sk = ax_scale(ax_head_max(k, hs), &ik), sv = ax_scale(ax_head_max(v, hs), &iv);
    if (li >= kvd) continue;
    const size_t row = (size_t)base[i] + t, at = row * kvd + li;
    ax_planes(k, sk, st.kh + at, st.kl + at);
    ax_planes(v, sv, st.vh + at, st.vl + at);
    if (li % hs == 0) {
      st.ks[(size_t)(li / hs) * st.rows + row] = ik;
      st.vs[(size_t)(li / hs) * st.rows + row] = iv;
    }
  }
}

__device__ __forceinline__ void ax_tmem_ld32(uint32_t taddr, uint32_t (&v)[32]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16, %17, %18, %19, "
      "%20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
      : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]), "=r"(v[8]), "=r"(v[9]),
        "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15]), "=r"(v[16]), "=r"(v[17]), "=r"(v[18]), "=r"(v[19]),
        "=r"(v[20]), "=r"(v[21]), "=r"(v[22]), "=r"(v[23]), "=r"(v[24]), "=r"(v[25]), "=r"(v[26]), "=r"(v[27]), "=r"(v[28]), "=r"(v[29]),
        "=r"(v[30]), "=r"(v[31])
      : "r"(taddr));
}
__device__ __forceinline__ void ax_tmem_st8(uint32_t taddr, const uint32_t (&v)[8]) {
  asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};"
               ::"r"(taddr), "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7]) : "memory");
}
// kind::f16, fp16 x fp16 -> fp32, M = 128, N = n, A and B K-major
__host__ __device__ constexpr uint32_t ax_idesc(int n) { return (1u << 4) | ((uint32_t)(n >> 3) << 17) | ((uint32_t)(128 >> 4) << 24); }
// D = A B + D 2^-11
__device__ __forceinline__ void ax_mma_over(uint32_t tmem_d, uint64_t adesc, uint64_t bdesc, uint32_t idesc) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.eq.b32 p, 0, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p, %4;\n\t}"
      ::"r"(tmem_d), "l"(adesc), "l"(bdesc), "r"(idesc), "n"(SPLIT_LO) : "memory");
}
__device__ __forceinline__ void ax_mma_ts_over(uint32_t tmem_d, uint32_t tmem_a, uint64_t bdesc, uint32_t idesc) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.eq.b32 p, 0, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p, %4;\n\t}"
      ::"r"(tmem_d), "r"(tmem_a), "l"(bdesc), "r"(idesc), "n"(SPLIT_LO) : "memory");
}
// MN-major B, SWIZZLE_128B: blocks of 64 columns x 8 rows of K; K groups 1024 bytes apart, column blocks 16 KB
__device__ __forceinline__ uint64_t ax_desc_mn(uint32_t saddr) {
  return (uint64_t)((saddr & 0x3FFFFu) >> 4) | (uint64_t)((128 * 128) >> 4) << 16 | (uint64_t)(1024 >> 4) << 32 | (uint64_t)1 << 46 | (uint64_t)2 << 61;
}

template <int HS>
__global__ void __launch_bounds__(256, HS == 64 ? 2 : 1)
attn_prefill_x3_kernel(const __grid_constant__ CUtensorMap mqh, const __grid_constant__ CUtensorMap mql, const __grid_constant__ CUtensorMap mkh,
                       const __grid_constant__ CUtensorMap mkl, const __grid_constant__ CUtensorMap mvh, const __grid_constant__ CUtensorMap mvl, const AttnX3P p) {
  constexpr int KBH = HS / 64;                       // 64-value blocks along the head
  constexpr int TILE = KBH * 128 * 128;              // a plane of a Q, K or V tile: [block][128 rows][128 bytes]
  constexpr int HH = HS / 2;                         // head columns per thread
  constexpr int TMEM_COLS = 256;                     // S (and P over it): 128 columns, P V: HS columns
  extern __shared__ unsigned char ax_raw[];
  __shared__ float s_max[2][AX_T];                   // row maxima / sums of the two column halves
  __shared__ float s_ks[2][AX_T], s_vs[2][AX_T];     // inverse scales of a tile's keys, of this tile and the next
  __shared__ float s_vp[2][AX_T], s_vm[2][4];        // largest of s_vs up to a key of the warp's 32, of all 32
  __shared__ uint64_t qbar, kbar, vbar, sbar, pbar;
  __shared__ uint32_t tmem_slot;
  __shared__ int abort_s, key_tiles;                 // key_tiles: of K, and of V, that are asked for; thread 0's
  unsigned char* smem = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(ax_raw) + 1023) & ~(uintptr_t)1023);
  unsigned char *Qs = smem, *Ks = smem + 2 * TILE, *Vs = smem + 4 * TILE;      // each hi | lo

  // warp w serves TMEM lanes 32 (w & 3) .. (query rows) and column half w >> 2
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int qd = warp & 3, hf = warp >> 2, row = qd * 32 + lane;
  const int tile = blockIdx.y, h = blockIdx.x;       // the longest tiles come first
  if (tid == 0) {
    tc_mbar_init(&qbar, 1); tc_mbar_init(&kbar, 1); tc_mbar_init(&vbar, 1); tc_mbar_init(&sbar, 1); tc_mbar_init(&pbar, 1);
    abort_s = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
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
  auto load = [&](unsigned char* dst, const CUtensorMap* hi, const CUtensorMap* lo, int col, int r, uint64_t* bar) {
    tc_mbar_expect_tx(bar, 2 * TILE);
#pragma unroll
    for (int kb = 0; kb < KBH; kb++) {
      tc_tma_2d(dst + kb * (128 * 128), hi, col + kb * 64, r, bar);
      tc_tma_2d(dst + TILE + kb * (128 * 128), lo, col + kb * 64, r, bar);
    }
  };
  auto scores = [&]() {
    constexpr uint32_t idesc = ax_idesc(AX_T);
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
#pragma unroll
    for (int part = 0; part < 3; part++) {           // lo.hi, hi.lo, hi.hi
#pragma unroll
      for (int kb = 0; kb < KBH; kb++) {
        const uint64_t a = tc_smem_desc(tc_smem_u32(Qs + (part == 0 ? TILE : 0) + kb * (128 * 128))), b = tc_smem_desc(tc_smem_u32(Ks + (part == 1 ? TILE : 0) + kb * (128 * 128)));
#pragma unroll
        for (int k = 0; k < 4; k++) {
          if (part == 2 && (kb | k) == 0) ax_mma_over(tmem_s, a, b, idesc);
          else tc_mma_f16(tmem_s, a + (uint64_t)(2 * k), b + (uint64_t)(2 * k), idesc, (uint32_t)((part | kb | k) != 0));
        }
      }
    }
    tc_commit(&sbar);
  };
  if (tid == 0) key_tiles = live_tile ? kmax / AX_T + 1 : 0;
  bool ok = true;
  if (warp == 0 && live_tile) {
    if (tc_elect()) {
      load(Qs, &mqh, &mql, h * HS, row0, &qbar);
      load(Ks, &mkh, &mkl, kh * HS, key_row0, &kbar);
      load(Vs, &mvh, &mvl, kh * HS, key_row0, &vbar);
      if (tc_mbar_wait(&qbar, 0u, abort_flag) && tc_mbar_wait(&kbar, 0u, abort_flag)) scores();
    }
    __syncwarp();
  }
  // inverse scales of the tile from key t0 on: threads 0 .. 127 K's, the others V's; 0 behind the last key
  const float* scales = (tid < AX_T ? p.ks : p.vs) + (size_t)kh * p.staged_rows + key_row0 + (tid & (AX_T - 1));
  auto scale_of = [&](int t0) { return t0 + (tid & (AX_T - 1)) <= kmax ? scales[t0] : 0.0f; };
  auto keep_scale = [&](float v, int buf) {
    if (tid < AX_T) {
      s_ks[buf][tid] = v;
    } else {
      s_vs[buf][tid - AX_T] = v;
      float m = v;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const float up = __shfl_up_sync(THA_FULL_MASK, m, o);
        if (lane >= o) m = fmaxf(m, up);
      }
      s_vp[buf][tid - AX_T] = m;
      if (lane == 31) s_vm[buf][qd] = m;
    }
  };
  keep_scale(scale_of(0), 0);
  __syncthreads();
  const int qrow = row < n ? row : n - 1, qpos = pos0 + qrow;
  // scores in units of log2(e): exp(x) = exp2(x * log2 e)
  const float qf = live_tile ? p.qs[(size_t)(row0 + qrow) * p.heads + h] * (1.4426950408889634f / sqrtf((float)HS)) : 0.0f;
  float m_run = -INFINITY, l_run = 0.0f;             // l_run: this thread's half of the row sum (both halves share m)
  float acc[HH];
#pragma unroll
  for (int c = 0; c < HH; c++) acc[c] = 0.0f;
  const uint32_t ts = tmem_s + ((uint32_t)(qd * 32) << 16) + (uint32_t)(64 * hf);
  const uint32_t tpv = tmem_pv + ((uint32_t)(qd * 32) << 16) + (uint32_t)(HH * hf);
  unsigned ph = 0;                                   // parity of this tile's phases
  for (int t0 = 0; t0 <= kmax; t0 += AX_T, ph ^= 1u) {
    const bool more = t0 + AX_T <= kmax, whole = t0 + AX_T - 1 <= pos0;   // whole: every row sees every key
    const float ahead = more ? scale_of(t0 + AX_T) : 0.0f;
    float c = 1.0f;                                  // a power of two from 2^-100 on; 1 for a row that sees no key of the tile
    if (const int seen = min(qpos - t0, AX_T - 1); seen >= 0) {
      c = s_vp[ph][seen];
#pragma unroll
      for (int x = 0; x < 3; x++)
        if (x < seen >> 5) c = fmaxf(c, s_vm[ph][x]);
    }
    const float up = 16384.0f / c;
    if (ok) ok = tc_mbar_wait(&sbar, ph, abort_flag);
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    if (warp == 0) {
      if (more && tc_elect()) load(Ks, &mkh, &mkl, kh * HS, key_row0 + t0 + AX_T, &kbar);
      __syncwarp();
    }
    // ---- softmax of this thread's half row (keys 64 hf .. 64 hf + 63 of the tile): the maximum first (exchanged with the other half through shared
    // memory), then, out of TMEM again, weights -> their planes over the scores that they came from: per 16 keys 8 columns of hi, 8 of lo
    const int tk = t0 + 64 * hf;                     // first key of this thread's columns
    float mt = -INFINITY;
#pragma unroll
    for (int half = 0; half < 2; half++) {
      uint32_t s[32];
      ax_tmem_ld32(ts + (uint32_t)(32 * half), s);
      asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
      for (int j = 0; j < 32; j += 4) {
        const float4 k4 = *reinterpret_cast<const float4*>(&s_ks[ph][64 * hf + 32 * half + j]);
        const float ks[4] = {k4.x, k4.y, k4.z, k4.w};
#pragma unroll
        for (int e = 0; e < 4; e++)
          if (whole || tk + 32 * half + j + e <= qpos) mt = fmaxf(mt, __uint_as_float(s[j + e]) * ks[e]);
      }
    }
    s_max[hf][row] = mt;
    __syncthreads();
    const float m_new = fmaxf(m_run, fmaxf(s_max[0][row], s_max[1][row]) * qf);   // finite: key 0 is visible to every row
    const float corr = exp2f(m_run - m_new);         // exp2(-inf) = 0 on the first tile
    float lsum = 0.0f;
#pragma unroll
    for (int x = 0; x < 4; x++) {                    // 16 keys at a time
      uint32_t s[16], hi[8], lo[8];
      tc_tmem_ld16(ts + (uint32_t)(16 * x), s);
      asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
      for (int j = 0; j < 16; j += 4) {
        const float4 k4 = *reinterpret_cast<const float4*>(&s_ks[ph][64 * hf + 16 * x + j]), v4 = *reinterpret_cast<const float4*>(&s_vs[ph][64 * hf + 16 * x + j]);
        const float ks[4] = {k4.x, k4.y, k4.z, k4.w}, vs[4] = {v4.x, v4.y, v4.z, v4.w};
        float w[4];
#pragma unroll
        for (int e = 0; e < 4; e++) {
          float pe = exp2f(fmaf(__uint_as_float(s[j + e]) * ks[e], qf, -m_new));
          if (!whole && tk + 16 * x + j + e > qpos) pe = 0.0f;
          lsum += pe;
          w[e] = pe;
        }
#pragma unroll
        for (int e = 0; e < 4; e += 2) split_f16x2(f32x2_mul(make_float2(w[e], w[e + 1]), make_float2(vs[e], vs[e + 1])), up, hi[(j + e) >> 1], lo[(j + e) >> 1]);
      }
      ax_tmem_st8(ts + (uint32_t)(16 * x), hi);
      ax_tmem_st8(ts + (uint32_t)(16 * x + 8), lo);
    }
    asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
    l_run = l_run * corr + lsum;
    m_run = m_new;
    if (more) keep_scale(ahead, ph ^ 1u);
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    // ---- P V: keys 16 x .. 16 x + 15; groups of 16 behind the tile's last key are left out
    if (warp == 0) {
      if (tc_elect() && tc_mbar_wait(&vbar, ph, abort_flag)) {
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        constexpr uint32_t idesc = ax_idesc(HS) | (1u << 16);
        const uint64_t vh = ax_desc_mn(tc_smem_u32(Vs)), vl = ax_desc_mn(tc_smem_u32(Vs + TILE));
        const int groups = more ? AX_T / 16 : (kmax - t0 + 16) / 16;
        for (int x = 0; x < groups; x++) {
          const uint32_t a = tmem_s + (uint32_t)(16 * x);
          tc_mma_f16_ts(tmem_pv, a + 8, vh + (uint64_t)(x * (2048 >> 4)), idesc, (uint32_t)(x != 0));
          tc_mma_f16_ts(tmem_pv, a, vl + (uint64_t)(x * (2048 >> 4)), idesc, 1u);
        }
        ax_mma_ts_over(tmem_pv, tmem_s, vh, idesc);
        for (int x = 1; x < groups; x++) tc_mma_f16_ts(tmem_pv, tmem_s + (uint32_t)(16 * x), vh + (uint64_t)(x * (2048 >> 4)), idesc, 1u);
        tc_commit(&pbar);
      }
      __syncwarp();
    }
    if (ok) ok = tc_mbar_wait(&pbar, ph, abort_flag);
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    if (warp == 0) {
      if (more && tc_elect()) {
        load(Vs, &mvh, &mvl, kh * HS, key_row0 + t0 + AX_T, &vbar);
        if (tc_mbar_wait(&kbar, ph ^ 1u, abort_flag)) scores();   // the next tile's, under this one's accumulator
      }
      __syncwarp();
    }
    const float f = c * (1.0f / 16384.0f);
#pragma unroll
    for (int c0 = 0; c0 < HH; c0 += 32) {
      uint32_t v[32];
      ax_tmem_ld32(tpv + (uint32_t)c0, v);
      asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
      for (int j = 0; j < 32; j++) acc[c0 + j] = fmaf(__uint_as_float(v[j]), f, acc[c0 + j] * corr);
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  }

  // ---- the row sum is the sum of its two halves; normalise and store this thread's half row
  __syncthreads();
  s_max[hf][row] = l_run;
  __syncthreads();
  if (live_tile && row < n && ok) {
    const float l = s_max[0][row] + s_max[1][row];
    float* orow = p.out + (size_t)(row0 + row) * p.dim + h * HS + HH * hf;
#pragma unroll
    for (int c = 0; c < HH; c += 4) *reinterpret_cast<float4*>(orow + c) = make_float4(acc[c] / l, acc[c + 1] / l, acc[c + 2] / l, acc[c + 3] / l);
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

bool attn_prefill_x3_supported(int head_size) { return head_size == 64 || head_size == 128; }

int x3_rope_launch(cudaStream_t st, bool pdl, int R, const float* part, int nz, long long zstride, int ld, const int* pos, int d, int kvd, int hs, const float* rc,
                   const float* rs, float* kc, float* vc, long long kv_bs, int loff, const int* slot, const KvPaged& pg, const X3Staged& staged) {
  THA_CUDA_OK(launch(x3_rope_kernel, dim3(ceil_div(ld / 4, 512), R), dim3(256), 0, st, pdl, part, nz, zstride, ld, pos, d, kvd, hs, rc, rs, kc, vc, kv_bs, loff, slot, pg, staged));
  return THA_STATUS_SUCCESS;
}

// kc, vc: the layer's slab (or the pool's base)
int x3_context_launch(cudaStream_t st, bool pdl, int n_seqs, int longest, const float* kc, const float* vc, long long kv_bs, const int* seq_slot, const int* upto,
                      const int* base, const KvPaged& pg, int kvd, int hs, const X3Staged& staged) {
  THA_CUDA_OK(launch(x3_context_kernel, dim3(ceil_div(kvd, 1024), longest < 4096 ? longest : 4096, n_seqs), dim3(256), 0, st, pdl, kc, vc, kv_bs, seq_slot, upto, base, pg, kvd,
                     hs, staged));
  return THA_STATUS_SUCCESS;
}

// tiles of up to 128 query rows, never across sequences, longest contexts first; a sequence's staged rows begin at its position 0, at a multiple of 128
int attn_prefill_x3_launch(cudaStream_t st, bool pdl, int n_tiles, int rows, int n_heads, int n_kv_heads, int head_size, float* out, const int* row_pos,
                           const int* tile_row0, const int* tile_n, const X3Staged& s) {
  if (!attn_prefill_x3_supported(head_size)) return THA_STATUS_NOT_SUPPORTED;
  const int d = n_heads * head_size, kvd = n_kv_heads * head_size;
  AttnX3P p;
  p.out = out; p.dim = d; p.kv_mul = n_heads / n_kv_heads; p.heads = n_heads; p.staged_rows = s.rows;
  p.qs = s.qs; p.ks = s.ks; p.vs = s.vs; p.row_pos = row_pos; p.row_stage = s.row; p.tile_row0 = tile_row0; p.tile_n = tile_n;
  THA_TRY_RC(gemm_tc_init(&p.error_flag));
  CUtensorMap m[6];
  THA_TRY_RC(tc_map(s.qh, rows, d, d, 128, &m[0], 2));
  THA_TRY_RC(tc_map(s.ql, rows, d, d, 128, &m[1], 2));
  THA_TRY_RC(tc_map(s.kh, s.rows, kvd, kvd, 128, &m[2], 2));
  THA_TRY_RC(tc_map(s.kl, s.rows, kvd, kvd, 128, &m[3], 2));
  THA_TRY_RC(tc_map(s.vh, s.rows, kvd, kvd, 128, &m[4], 2));
  THA_TRY_RC(tc_map(s.vl, s.rows, kvd, kvd, 128, &m[5], 2));
  const size_t smem = (size_t)6 * head_size * 256 + 1024;
  auto k = head_size == 64 ? attn_prefill_x3_kernel<64> : attn_prefill_x3_kernel<128>;
  THA_CUDA_OK(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  THA_CUDA_OK(launch(k, dim3(n_heads, n_tiles), dim3(256), smem, st, pdl, m[0], m[1], m[2], m[3], m[4], m[5], p));
  return THA_STATUS_SUCCESS;
}

}  // namespace tha
