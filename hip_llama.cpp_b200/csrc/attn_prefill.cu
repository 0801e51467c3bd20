// Causal attention for batched prompt ingestion: many query rows of one sequence against its
// KV cache in one pass (the decode kernel of attention.cu reads the whole prefix once per row,
// which is quadratic in traffic for a long prompt).
//
// Same arithmetic as the reference's per-position loop (run.cc:288-321: score = q.k / sqrt(hs),
// softmax over t <= pos, weighted sum of V) evaluated tile by tile with an online softmax, all of it in fp32:
//   CTA = 16 RI consecutive query rows (64 or 128) of one (sequence, head); loop over 64-key tiles of the cache
//   (which already holds this layer's K/V rows of the chunk -- tc_rope_scatter_kernel ran first);
//   S = Q K^T on an RI x 4 register micro-tile per thread (rows ty + 16 i, keys tx + 16 j, four channels per 128-bit
//   shared-memory read), running max / sum per row, P staged in shared memory, O += P V.
// K and V tiles arrive by cp.async, whole rows at a time: V of a tile while its scores are computed, K of the next one under P V -- one
// buffer each and two barriers per tile.  Bound by fp32 FMA (128 per SM and clock) and the shared-memory reads beside
// it: per 16 FMAs 1.5 of 128 bits in Q K^T and 1.0 (heads of 128) or 1.5 (of 64) in P V at RI = 8; 2, 1.5 and 2 at RI = 4.
// The longest tiles start first.  Q8_0 prompts, and fp32 ones that attn_prefill_x3.cu's rule leaves or whose planes get no scratch.
#include "common.cuh"
#include "workspace.h"

namespace tha {

struct AttnPrefillP {
  const float* q; float* out; float* out_hi; float* out_lo;   // [rows, dim]
  const float* kc; const float* vc;                           // cache base of the layer
  long long kv_batch_stride; int kv_dim, kv_mul, dim;
  const int* row_slot; const int* row_pos;                    // [rows]
  const int* tile_row0; const int* tile_n;                    // [tiles]: first row and row count (<= 16 RI) of each query tile
  KvPaged pg;                                                 // pg.table != nullptr: kc / vc are block pools, rows found through the table
};

constexpr int PF_TK = 64, PF_PS = PF_TK + 4;   // keys per tile, row pitch of P

__device__ __forceinline__ float pf_tf32(float v) { return __uint_as_float((__float_as_uint(v) + 0x1000u) & 0xFFFFE000u); }
__device__ __forceinline__ void pf_cp16(float* dst, const float* src, bool live) {   // 16 bytes, zeros where the key is past the end
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src), "r"(live ? 16 : 0) : "memory");
}

template <int HS, int RI>
constexpr size_t pf_smem() { return ((size_t)(16 * RI + PF_TK) * (HS + 4) + (size_t)PF_TK * HS + (size_t)16 * RI * PF_PS) * sizeof(float); }

template <int HS, int RI>
__global__ void __launch_bounds__(256) attn_prefill_kernel(const AttnPrefillP p) {
  constexpr int TQ = 16 * RI, KS = HS + 4;   // rows pitched by 4 banks: conflict-free 128-bit reads of 16 neighbouring rows
  constexpr int CW = HS / 16;              // output columns per thread
  constexpr int NV = (CW >= 4) ? CW / 4 : 1;
  constexpr int VW = (CW >= 4) ? 4 : CW;   // floats per V read
  extern __shared__ float4 pf_smem4[];
  float* Qs = reinterpret_cast<float*>(pf_smem4);   // [TQ][KS]
  float* Ks = Qs + TQ * KS;                          // [64][KS]
  float* Vs = Ks + PF_TK * KS;                       // [64][HS]
  float* Ps = Vs + PF_TK * HS;                       // [TQ][PF_PS]

  pdl_wait();
  pdl_trigger();
  const int heads = p.dim / HS, tile = blockIdx.x / heads, h = blockIdx.x - tile * heads;   // the heads of a tile side by side
  const int row0 = p.tile_row0[tile], n = p.tile_n[tile];
  const int slot = p.row_slot[row0], pos0 = p.row_pos[row0];
  if (pos0 < 0 || n <= 0) return;
  const int tid = threadIdx.x, tx = tid & 15, ty = tid >> 4;
  const int kh = h / p.kv_mul;
  const float* kbase = (p.pg.table ? p.kc : p.kc + (size_t)slot * p.kv_batch_stride) + kh * HS;
  const float* vbase = (p.pg.table ? p.vc : p.vc + (size_t)slot * p.kv_batch_stride) + kh * HS;
  const int kmax = pos0 + n - 1;   // last key any row of the tile may see
  const float sqrt_hs = sqrtf((float)HS);
  constexpr int C4 = HS / 4;       // float4 per row

  // keys tk0 .. tk0 + 63 -> dst (row pitch `pitch`): consecutive threads take consecutive 16-byte pieces of a row
  auto load_rows = [&](float* dst, int pitch, const float* base, int tk0) {
#pragma unroll
    for (int i0 = 0; i0 < PF_TK * C4; i0 += 256) {
      const int i = i0 + tid, r = i / C4, c = i - r * C4;
      const int t = tk0 + r;
      const bool live = t <= kmax;
      const int tr = live ? t : kmax;
      const long long roff = p.pg.table ? kv_paged_off(p.pg, slot, tr, p.kv_dim) : (long long)tr * p.kv_dim;
      pf_cp16(dst + r * pitch + 4 * c, base + roff + 4 * c, live);
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  static_assert(PF_TK * C4 % 256 == 0, "every thread copies the same number of pieces");
  load_rows(Ks, KS, kbase, 0);
  for (int i = tid; i < TQ * C4; i += 256) {
    const int r = i / C4, c = i - r * C4;
    *reinterpret_cast<float4*>(Qs + r * KS + 4 * c) = *reinterpret_cast<const float4*>(p.q + (size_t)(row0 + (r < n ? r : n - 1)) * p.dim + h * HS + 4 * c);
  }

  float m[RI], l[RI], o[RI][CW];
  int qpos[RI];
#pragma unroll
  for (int i = 0; i < RI; i++) {
    m[i] = -INFINITY; l[i] = 0.0f;
    const int r = ty + 16 * i;
    qpos[i] = pos0 + ((r < n) ? r : n - 1);
#pragma unroll
    for (int c = 0; c < CW; c++) o[i][c] = 0.0f;
  }

  for (int tk0 = 0; tk0 <= kmax; tk0 += PF_TK) {
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    __syncthreads();   // this tile's K is in place (and Q, the first time); the previous tile's V and P are no longer read
    load_rows(Vs, HS, vbase, tk0);

    // ---- S = Q K^T : rows ty + 16 i, keys tx + 16 j ----
    float s[RI][4];
#pragma unroll
    for (int i = 0; i < RI; i++)
#pragma unroll
      for (int j = 0; j < 4; j++) s[i][j] = 0.0f;
#pragma unroll 2
    for (int k = 0; k < HS; k += 4) {
      float4 b[4];
#pragma unroll
      for (int j = 0; j < 4; j++) b[j] = *reinterpret_cast<const float4*>(Ks + (tx + 16 * j) * KS + k);
#pragma unroll
      for (int i = 0; i < RI; i++) {
        const float4 a = *reinterpret_cast<const float4*>(Qs + (ty + 16 * i) * KS + k);
#pragma unroll
        for (int j = 0; j < 4; j++) s[i][j] = dot4(a, b[j], s[i][j]);
      }
    }
    // ---- scale, causal mask, online softmax (row statistics shared by the 16 threads of a row) ----
#pragma unroll
    for (int i = 0; i < RI; i++) {
      float rmax = -INFINITY;
#pragma unroll
      for (int j = 0; j < 4; j++) {
        const int t = tk0 + tx + 16 * j;
        s[i][j] = (t <= qpos[i]) ? s[i][j] / sqrt_hs : -INFINITY;
        rmax = fmaxf(rmax, s[i][j]);
      }
#pragma unroll
      for (int off = 8; off > 0; off >>= 1) rmax = fmaxf(rmax, __shfl_xor_sync(THA_FULL_MASK, rmax, off));
      const float mn = fmaxf(m[i], rmax);          // finite: key 0 is visible to every row in the first tile
      const float corr = expf(m[i] - mn);          // exp(-inf) = 0 on the first tile
#pragma unroll
      for (int j = 0; j < 4; j++) {
        s[i][j] = expf(s[i][j] - mn);
        Ps[(ty + 16 * i) * PF_PS + tx + 16 * j] = s[i][j];
      }
      // partial of the row sum, reduced at the end: thread tx adds the four neighbouring keys 4 m .. 4 m + 3, m = 4 (tx & 3) + (tx >> 2), which four
      // neighbouring threads hold (three exchanges).  The grouping is part of the result's bits: a quantiser behind it turns a last bit into
      // a step, and with sums in another order 3 of 79 next tokens of quantised prompts changed.
      const bool b0 = tx & 1, b1 = tx & 2;
      const float u0 = (b0 ? s[i][1] : s[i][0]) + __shfl_xor_sync(THA_FULL_MASK, b0 ? s[i][0] : s[i][1], 1);   // column j = tx & 1
      const float u1 = (b0 ? s[i][3] : s[i][2]) + __shfl_xor_sync(THA_FULL_MASK, b0 ? s[i][2] : s[i][3], 1);   // and that plus two
      l[i] = l[i] * corr + ((b1 ? u1 : u0) + __shfl_xor_sync(THA_FULL_MASK, b1 ? u0 : u1, 2));
#pragma unroll
      for (int c = 0; c < CW; c++) o[i][c] *= corr;
      m[i] = mn;
    }
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    __syncthreads();   // V and P are in place, every score is computed: K's buffer is free
    if (tk0 + PF_TK <= kmax) load_rows(Ks, KS, kbase, tk0 + PF_TK);

    // ---- O += P V : rows ty + 16 i, columns tx*VW + 64*v ----
#pragma unroll 1
    for (int t = 0; t < PF_TK; t += 4) {
      float4 pr[RI];
#pragma unroll
      for (int i = 0; i < RI; i++) pr[i] = *reinterpret_cast<const float4*>(Ps + (ty + 16 * i) * PF_PS + t);
#pragma unroll
      for (int tt = 0; tt < 4; tt++) {
        float vv[CW];
        const float* vr = Vs + (t + tt) * HS;
        if constexpr (VW == 4) {
#pragma unroll
          for (int v = 0; v < NV; v++) {
            const float4 a = *reinterpret_cast<const float4*>(vr + tx * 4 + 64 * v);
            vv[4 * v + 0] = a.x; vv[4 * v + 1] = a.y; vv[4 * v + 2] = a.z; vv[4 * v + 3] = a.w;
          }
        } else {
#pragma unroll
          for (int c = 0; c < CW; c++) vv[c] = vr[tx * CW + c];
        }
#pragma unroll
        for (int i = 0; i < RI; i++) {
          const float w = tt == 0 ? pr[i].x : (tt == 1 ? pr[i].y : (tt == 2 ? pr[i].z : pr[i].w));
#pragma unroll
          for (int c = 0; c < CW; c++) o[i][c] = fmaf(w, vv[c], o[i][c]);
        }
      }
    }
  }

  // ---- normalise and store (fp32 row and its tf32 hi/lo split for the wo matmul) ----
#pragma unroll
  for (int i = 0; i < RI; i++) {
    float L = l[i];
    L += __shfl_xor_sync(THA_FULL_MASK, L, 2);   // m ^ 8, m ^ 4, m ^ 2, m ^ 1
    L += __shfl_xor_sync(THA_FULL_MASK, L, 1);
    L += __shfl_xor_sync(THA_FULL_MASK, L, 8);
    L += __shfl_xor_sync(THA_FULL_MASK, L, 4);
    const int r = ty + 16 * i;
    if (r >= n) continue;
    const size_t base = (size_t)(row0 + r) * p.dim + h * HS;
#pragma unroll
    for (int v = 0; v < CW / VW; v++) {
      const int col = (VW == 4) ? tx * 4 + 64 * v : tx * CW;
      float hi[VW], val[VW];
#pragma unroll
      for (int e = 0; e < VW; e++) { val[e] = o[i][v * VW + e] / L; hi[e] = pf_tf32(val[e]); }
      if constexpr (VW == 4) {
        *reinterpret_cast<float4*>(p.out + base + col) = make_float4(val[0], val[1], val[2], val[3]);
        if (p.out_hi) {
          *reinterpret_cast<float4*>(p.out_hi + base + col) = make_float4(hi[0], hi[1], hi[2], hi[3]);
          *reinterpret_cast<float4*>(p.out_lo + base + col) = make_float4(val[0] - hi[0], val[1] - hi[1], val[2] - hi[2], val[3] - hi[3]);
        }
      } else {
#pragma unroll
        for (int e = 0; e < VW; e++) {
          p.out[base + col + e] = val[e];
          if (p.out_hi) { p.out_hi[base + col + e] = hi[e]; p.out_lo[base + col + e] = val[e] - hi[e]; }
        }
      }
    }
  }
}

bool attn_prefill_supported(int head_size, int kv_dim) {
  return (head_size == 16 || head_size == 32 || head_size == 64 || head_size == 128) && kv_dim % 4 == 0;
}
// Query rows per tile (the result's bits do not depend on it): 128, with a quarter to a third fewer shared-memory reads per FMA, where the prompts fill
// such tiles and these (tiles128 x heads of them) leave no SM without one for long, 64 otherwise.  us a prefill with tiles of 64 / 128: 32 heads of
// 128, one prompt of 256 890 / 933, of 512 1683 / 1754, of 640 2102 / 2144 (Q8_0; 160 tiles of 128), four of 256 4557 / 4529 (fp32; 256); 12 heads
// of 64, eight prompts of 192 2315 / 2455 (192), one of 512 1776 / 1738 (48).
int attn_prefill_tile_rows(int rows, int n_seqs, int tiles128, int heads) { return rows >= 192 * n_seqs && tiles128 * heads >= 256 ? 128 : 64; }

// tile_row0 / tile_n: tiles of at most tile_rows (64 or 128) query rows, never across sequences, longest contexts first
int attn_prefill_launch(cudaStream_t stream, int n_tiles, int n_heads, int n_kv_heads, int head_size, const float* q,
                        float* out, float* out_hi, float* out_lo, const float* kc, const float* vc,
                        long long kv_batch_stride, const int* row_slot, const int* row_pos, const int* tile_row0,
                        const int* tile_n, bool pdl, const KvPaged* pg, int tile_rows) {
  if (!attn_prefill_supported(head_size, n_kv_heads * head_size) || (tile_rows != 64 && tile_rows != 128)) return THA_STATUS_NOT_SUPPORTED;
  AttnPrefillP p;
  p.q = q; p.out = out; p.out_hi = out_hi; p.out_lo = out_lo; p.kc = kc; p.vc = vc;
  if (pg) p.pg = *pg; else p.pg = KvPaged{};
  p.kv_batch_stride = kv_batch_stride; p.kv_dim = n_kv_heads * head_size; p.kv_mul = n_heads / n_kv_heads;
  p.dim = n_heads * head_size;
  p.row_slot = row_slot; p.row_pos = row_pos; p.tile_row0 = tile_row0; p.tile_n = tile_n;
  void (*k)(const AttnPrefillP) = nullptr;
  size_t smem = 0;
  const bool big = tile_rows == 128;
  switch (head_size) {
    case 16: k = big ? attn_prefill_kernel<16, 8> : attn_prefill_kernel<16, 4>; smem = big ? pf_smem<16, 8>() : pf_smem<16, 4>(); break;
    case 32: k = big ? attn_prefill_kernel<32, 8> : attn_prefill_kernel<32, 4>; smem = big ? pf_smem<32, 8>() : pf_smem<32, 4>(); break;
    case 64: k = big ? attn_prefill_kernel<64, 8> : attn_prefill_kernel<64, 4>; smem = big ? pf_smem<64, 8>() : pf_smem<64, 4>(); break;
    default: k = big ? attn_prefill_kernel<128, 8> : attn_prefill_kernel<128, 4>; smem = big ? pf_smem<128, 8>() : pf_smem<128, 4>(); break;
  }
  if (smem > 40 * 1024) THA_CUDA_OK(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  THA_CUDA_OK(launch(k, dim3((unsigned)n_tiles * n_heads), dim3(256), smem, stream, pdl, p));
  return THA_STATUS_SUCCESS;
}

}  // namespace tha
