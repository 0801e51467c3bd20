// Softmax attention of single rows (decoding: a sequence with one row in the step) of the layer-program path, in fp32 straight from the cache rows.
//
// Which form a row takes depends on its own sequence alone: a decoded token is computed here whether or not another sequence brings a prompt
// portion to the same step (the tiled kernels, which round to bf16 in that number format, then take the longer portions only).  What still
// depends on the step is the number of runs a context is cut into, the order of an fp32 sum.
// The tiled kernels (hybrid_ops.cu) give a block 16 to 128 (position, head) pairs and stage key tiles through shared memory; with
// one position per sequence most pairs are empty and a block walks its tiles one load latency after the other.  Here a block takes one row,
// up to four query heads of one key/value head, and a run of 32-key tiles.  Eight lanes share a key (a lane: four channels of every 32), so
// a warp's load instruction covers four keys' rows; of a tile each of the four warps takes eight keys, all of whose K and V loads are in
// flight at once; the running maximum, sum and accumulator live in registers per group of eight lanes and meet only at the end of
// the run.  Nothing is rounded: q, keys, values and weights stay fp32 in both number formats.
// Bound by the latency of a run's loads, and by the cache rows it reads where there are many.
#include "common.cuh"
#include "hybrid_ops.cuh"

namespace tha {

constexpr int AR_HEADS = 4, AR_MAXD = 128, AR_THREADS = 128;

__device__ __forceinline__ float4 ar_ld(const float* p) { return ldg_stream(reinterpret_cast<const float4*>(p)); }

template <typename T, int GS>
__global__ void __launch_bounds__(AR_THREADS) hyb_attn_row_kernel(tha_attn_t a, tha_rows_t rows, tha_kv_t kv, const float* __restrict__ q, T* __restrict__ out,
                                                                  int splits, float* __restrict__ partial, const float* __restrict__ gate, long long ldg) {
  hyb_pdl_enter();
  constexpr int NI = AR_MAXD / 32;                 // float4 per lane of a row of up to 128 channels
  __shared__ float sm_acc[4][GS][AR_MAXD];
  __shared__ float sm_ml[4][GS][2];
  const int D = a.dim, E = a.vdim, gsize = a.heads / a.kv_heads;
  const int seq = blockIdx.x / splits, sp = blockIdx.x - seq * splits, g = blockIdx.y, h0 = blockIdx.z * GS;
  const int r = rows.seq_first[seq];
  if (rows.seq_first[seq + 1] - r != 1) return;   // a longer portion: the tiled kernels'
  const int gv = a.v_share > 1 ? g / a.v_share : g;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, kq = lane >> 3, c4 = 4 * (lane & 7);
  const int p = rows.pos[r], slot = rows.seq_slot[seq];
  const int first = a.chunk > 0 ? (p / a.chunk) * a.chunk : 0;
  float4 qv[GS][NI], acc[GS][NI];
  float m_run[GS], l_run[GS], hs[GS];
#pragma unroll
  for (int h = 0; h < GS; h++) {
    const int hg = h0 + h;
    const float* qr = q + ((size_t)r * a.heads + (size_t)g * gsize + (hg < gsize ? hg : 0)) * D;
    hs[h] = a.head_scale ? a.head_scale[g * gsize + (hg < gsize ? hg : 0)] : 1.0f;
    m_run[h] = -INFINITY; l_run[h] = 0.f;
#pragma unroll
    for (int i = 0; i < NI; i++) {
      acc[h][i] = make_float4(0.f, 0.f, 0.f, 0.f);
      qv[h][i] = 32 * i < D ? *reinterpret_cast<const float4*>(qr + 32 * i + c4) : make_float4(0.f, 0.f, 0.f, 0.f);
    }
  }
  const HybTiles tiles = hyb_attn_tiles(a, first, p, p);
  const int per = (tiles.n + splits - 1) / splits, ti_end = min(tiles.n, (sp + 1) * per);
  for (int ti = sp * per; ti < ti_end; ti++) {
    const int kt = (ti < tiles.n_a ? tiles.begin + 32 * ti : tiles.resume + 32 * (ti - tiles.n_a)) + 8 * warp;
    // this warp's eight keys: lanes 0..7 look their rows up, key 4 j + kq then goes to lanes kq * 8 ..
    const int mine = kt + (lane & 7);
    const size_t row = (mine <= p && mine >= first) ? hyb_kv_row(kv, slot, mine, a.cache_layer) : (size_t)-1;
    float4 kr[2][NI], vr[2][NI];
    bool vis[2];
#pragma unroll
    for (int j = 0; j < 2; j++) {
      const size_t at = __shfl_sync(THA_FULL_MASK, row, 4 * j + kq);
      vis[j] = at != (size_t)-1 && hyb_attn_sees(a, kt + 4 * j + kq, p, first);
      const float *kp = kv.k_pool + (vis[j] ? at : 0) + (size_t)g * D + c4, *vp = kv.v_pool + (vis[j] ? at : 0) + (size_t)gv * E + c4;
#pragma unroll
      for (int i = 0; i < NI; i++) kr[j][i] = vis[j] && 32 * i < D ? ar_ld(kp + 32 * i) : make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
      for (int i = 0; i < NI; i++) vr[j][i] = vis[j] && 32 * i < E ? ar_ld(vp + 32 * i) : make_float4(0.f, 0.f, 0.f, 0.f);
    }
#pragma unroll
    for (int h = 0; h < GS; h++) {
      float s[2];
#pragma unroll
      for (int j = 0; j < 2; j++) {
        float d = 0.f;
#pragma unroll
        for (int i = 0; i < NI; i++) d = dot4(qv[h][i], kr[j][i], d);
        d += __shfl_xor_sync(THA_FULL_MASK, d, 1);
        d += __shfl_xor_sync(THA_FULL_MASK, d, 2);
        d += __shfl_xor_sync(THA_FULL_MASK, d, 4);
        d = d * a.scale * hs[h];
        if (a.softcap > 0.f) d = hyb_softcap(d, a.softcap);
        if (a.rel && vis[j] && h0 + h < gsize) d += hyb_attn_rel(a, g * gsize + h0 + h, p - (kt + 4 * j + kq));
        s[j] = vis[j] ? d : -INFINITY;
      }
      const float m_new = fmaxf(m_run[h], fmaxf(s[0], s[1]));
      if (m_new > -INFINITY) {
        const float corr = expf(m_run[h] - m_new), w0 = expf(s[0] - m_new), w1 = expf(s[1] - m_new);
        l_run[h] = l_run[h] * corr + (w0 + w1);
        m_run[h] = m_new;
#pragma unroll
        for (int i = 0; i < NI; i++) {
          acc[h][i].x = fmaf(w1, vr[1][i].x, fmaf(w0, vr[0][i].x, acc[h][i].x * corr));
          acc[h][i].y = fmaf(w1, vr[1][i].y, fmaf(w0, vr[0][i].y, acc[h][i].y * corr));
          acc[h][i].z = fmaf(w1, vr[1][i].z, fmaf(w0, vr[0][i].z, acc[h][i].z * corr));
          acc[h][i].w = fmaf(w1, vr[1][i].w, fmaf(w0, vr[0][i].w, acc[h][i].w * corr));
        }
      }
    }
  }
  // the four key groups of a warp, then the four warps
#pragma unroll
  for (int h = 0; h < GS; h++) {
    float M = fmaxf(m_run[h], __shfl_xor_sync(THA_FULL_MASK, m_run[h], 8));
    M = fmaxf(M, __shfl_xor_sync(THA_FULL_MASK, M, 16));
    const float f = m_run[h] > -INFINITY ? expf(m_run[h] - M) : 0.f;
    float l = l_run[h] * f;
    l += __shfl_xor_sync(THA_FULL_MASK, l, 8);
    l += __shfl_xor_sync(THA_FULL_MASK, l, 16);
#pragma unroll
    for (int i = 0; i < NI; i++) {
      float v[4] = {acc[h][i].x * f, acc[h][i].y * f, acc[h][i].z * f, acc[h][i].w * f};
#pragma unroll
      for (int e = 0; e < 4; e++) {
        v[e] += __shfl_xor_sync(THA_FULL_MASK, v[e], 8);
        v[e] += __shfl_xor_sync(THA_FULL_MASK, v[e], 16);
      }
      if (kq == 0) *reinterpret_cast<float4*>(&sm_acc[warp][h][32 * i + c4]) = make_float4(v[0], v[1], v[2], v[3]);
    }
    if (lane == 0) { sm_ml[warp][h][0] = M; sm_ml[warp][h][1] = l; }
  }
  __syncthreads();
#pragma unroll 1
  for (int h = warp; h < GS; h += 4) {
    if (h0 + h >= gsize) break;
    const int head = g * gsize + h0 + h;
    float M = -INFINITY, L = 0.f, w[4];
#pragma unroll
    for (int x = 0; x < 4; x++) M = fmaxf(M, sm_ml[x][h][0]);
#pragma unroll
    for (int x = 0; x < 4; x++) { w[x] = sm_ml[x][h][0] > -INFINITY ? expf(sm_ml[x][h][0] - M) : 0.f; L += w[x] * sm_ml[x][h][1]; }
    const float inv = splits > 1 ? 1.0f : hyb_attn_final_factor(a, head, M, L, gate ? gate + (size_t)r * ldg : nullptr);
    float* pd = splits > 1 ? partial + (((size_t)sp * rows.n_seqs + seq) * a.heads + head) * (E + 2) : nullptr;
    for (int e = lane; e < E; e += 32) {
      float o = 0.f;
#pragma unroll
      for (int x = 0; x < 4; x++) o += w[x] * sm_acc[x][h][e];
      const size_t at = ((size_t)r * a.heads + head) * E + e;
      if (pd) pd[e] = o;
      else if (a.out_f32) reinterpret_cast<float*>(out)[at] = o * inv;
      else hyb_store(out + at, o * inv);
    }
    if (pd && lane == 0) { pd[E] = M; pd[E + 1] = L; }
  }
}

// Heads of 32, 64, 96 or 128 channels on 16-byte aligned cache rows; groups of more than eight query heads fill the
// tiled kernels' pairs, and here their key rows would be read a third time.
bool hyb_attn_row_ok(const tha_attn_t* a, const tha_kv_t* kv, const float* q) {
  return a->heads <= 2 * AR_HEADS * a->kv_heads && a->dim % 32 == 0 && a->vdim % 32 == 0 && a->dim <= AR_MAXD && a->vdim <= AR_MAXD &&
         kv->kv_dim % 4 == 0 && aligned16(kv->k_pool) && aligned16(kv->v_pool) && aligned16(q);
}
// Runs of a row's key tiles, were every sequence a single row: blocks for two to four on an SM, two tiles each (the number rounded up: rounded down, most
// contexts had runs of three tiles, one after the other.  Two layers of 16 heads on 4, 2 requests at 180 .. 560: 193 -> 187 us a step).
int hyb_attn_row_splits(const tha_attn_t* a, const tha_rows_t* rows, int max_keys) {
  const int gsize = a->heads / a->kv_heads;
  const long long blocks = (long long)rows->n_seqs * a->kv_heads * ceil_div(gsize, AR_HEADS);
  long long s = ceil_div(4 * 148, (int)(blocks < 4 * 148 ? blocks : 4 * 148));
  const int most = (max_keys + 63) / 64;
  if (s > most) s = most;
  return s < 1 ? 1 : (s > 32 ? 32 : (int)s);
}
template <typename T>
static int row_launch(cudaStream_t s, const tha_attn_t* a, const tha_rows_t* rows, const tha_kv_t* kv, const float* q, T* out, int splits, float* partial,
                      const float* gate, long long ldg) {
  const int gsize = a->heads / a->kv_heads, gs = gsize >= 3 ? AR_HEADS : gsize;
  const dim3 grid(rows->n_seqs * splits, a->kv_heads, ceil_div(gsize, gs));
  if (gs == 1) THA_CUDA_OK(launch(hyb_attn_row_kernel<T, 1>, grid, dim3(AR_THREADS), 0, s, pdl_enabled() != 0, *a, *rows, *kv, q, out, splits, partial, gate, ldg));
  else if (gs == 2) THA_CUDA_OK(launch(hyb_attn_row_kernel<T, 2>, grid, dim3(AR_THREADS), 0, s, pdl_enabled() != 0, *a, *rows, *kv, q, out, splits, partial, gate, ldg));
  else THA_CUDA_OK(launch(hyb_attn_row_kernel<T, AR_HEADS>, grid, dim3(AR_THREADS), 0, s, pdl_enabled() != 0, *a, *rows, *kv, q, out, splits, partial, gate, ldg));
  return THA_STATUS_SUCCESS;
}
int hyb_attn_row_launch(cudaStream_t s, int dtype, const tha_attn_t* a, const tha_rows_t* rows, const tha_kv_t* kv, const float* q, void* out, int splits,
                        float* partial, const float* gate, long long ldg) {
  return dtype == THA_DT_BF16 ? row_launch(s, a, rows, kv, q, (__nv_bfloat16*)out, splits, partial, gate, ldg)
                              : row_launch(s, a, rows, kv, q, (float*)out, splits, partial, gate, ldg);
}
}  // namespace tha
