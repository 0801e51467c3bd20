// Softmax attention of single rows (decoding: a sequence with one row in the step) of the layer-program path, in fp32 straight from the cache rows.
//
// Which form a row takes depends on its own sequence alone: a decoded token is computed here whether or not another sequence brings a prompt
// portion to the same step (the tiled kernels, which round to bf16 in that number format, then take the longer portions only).  What still
// depends on the step is the number of runs a context is cut into, the order of an fp32 sum.
// The tiled kernels (hybrid_ops.cu) give a block 16 to 128 (position, head) pairs and stage key tiles through shared memory; with
// one position per sequence most pairs are empty and a block walks its tiles one load latency after the other.  Here a block takes one row,
// up to four query heads of one key/value head, and a run of 32-key tiles.  Of a tile each of the four warps takes eight keys and copies their
// rows to a ring of three tiles in shared memory of its own (cp.async), so that a usual run is in flight at once; eight lanes share a key (a lane:
// four channels of every 32); the running maximum, sum and accumulator live in registers per group of eight lanes and meet only at the end of
// the run.  Nothing is rounded: q, keys, values and weights stay fp32 in both number formats.
// Inside a step of single rows all keys but those that the step itself writes are there before the kernel ahead is done, so they are asked for ahead of
// the wait for it.  What the step writes is one row a sequence: the row's own key, and the key of another sequence where a caller gives two of them one slot or one
// block.  The distance bias is asked for with a tile and not score by score.
// Bound by the latency of what follows that wait (q, the newest key, three tiles' arithmetic, the meeting of the warps), and by the cache rows it
// reads where there are many.  16 heads on 4 of 128 channels, 2 rows at 1100 .. 2900, behind the kernel ahead: tiles loaded to registers one by
// one 15.2 us; the ring, ahead of the wait 11.4; the bias with the tile 9.0; all heads' scores before their sums 8.4.
#include "common.cuh"
#include "hybrid_ops.cuh"

namespace tha {

constexpr int AR_HEADS = 4, AR_MAXD = 128, AR_THREADS = 128;
constexpr int AR_STAGES = 3;   // tiles of a run in flight

// sixteen bytes from global to shared memory behind the thread's back; bytes 0: zeros, src is not read
__device__ __forceinline__ void ar_copy16(void* dst, const float* src, int bytes) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src), "r"(bytes) : "memory");
}
__device__ __forceinline__ void ar_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void ar_await() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

template <typename T, int GS>
__global__ void __launch_bounds__(AR_THREADS) hyb_attn_row_kernel(tha_attn_t a, tha_rows_t rows, tha_kv_t kv, const float* q, T* __restrict__ out,
                                                                  int splits, float* __restrict__ partial, const float* gate, long long ldg, int early) {
  pdl_trigger();
  if (!early) pdl_wait();
  constexpr int NI = AR_MAXD / 32;                 // float4 per lane of a row of up to 128 channels
  extern __shared__ __align__(16) float ar_ring[];
  __shared__ float sm_acc[4][GS][AR_MAXD];
  __shared__ float sm_ml[4][GS][2];
  const int D = a.dim, E = a.vdim, gsize = a.heads / a.kv_heads;
  const int seq = blockIdx.x / splits, sp = blockIdx.x - seq * splits, g = blockIdx.y, h0 = blockIdx.z * GS;
  const int r = rows.seq_first[seq];
  if (rows.seq_first[seq + 1] - r != 1) {         // a longer portion: the tiled kernels'
    if (early) pdl_wait();                         // no kernel ends ahead of the one before it
    return;
  }
  const int gv = a.v_share > 1 ? g / a.v_share : g;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, kq = lane >> 3, c4 = 4 * (lane & 7);
  const int p = rows.pos[r], slot = rows.seq_slot[seq];
  const int first = a.chunk > 0 ? (p / a.chunk) * a.chunk : 0;
  const HybTiles tiles = hyb_attn_tiles(a, first, p, p);
  const int per = (tiles.n + splits - 1) / splits, ti0 = sp * per, ti_end = min(tiles.n, ti0 + per);
  auto tile_key = [&](int ti) { return (ti < tiles.n_a ? tiles.begin + 32 * ti : tiles.resume + 32 * (ti - tiles.n_a)) + 8 * warp; };
  // cache row of this lane's key (lane & 7) of the warp's eight of a tile
  auto row_of = [&](int ti) {
    const int mine = tile_key(ti) + (lane & 7);
    return (mine <= p && mine >= first) ? hyb_kv_row(kv, slot, mine, a.cache_layer) : (size_t)-1;
  };
  // those keys that `take` has a bit of on their way to the tile's place in the ring: key 4 j + kq goes to lanes kq * 8 ..
  float* ring = ar_ring + (size_t)warp * AR_STAGES * 8 * (D + E);
  auto fetch = [&](int ti, size_t row, unsigned take) {
    const int kt = tile_key(ti);
    float* st = ring + (size_t)((ti - ti0) % AR_STAGES) * 8 * (D + E);
#pragma unroll
    for (int j = 0; j < 2; j++) {
      const int key = kt + 4 * j + kq;
      const size_t at = __shfl_sync(THA_FULL_MASK, row, 4 * j + kq);
      if (!(take >> (4 * j + kq) & 1u)) continue;
      const bool vis = at != (size_t)-1 && hyb_attn_sees(a, key, p, first);
      const float *kp = kv.k_pool + (vis ? at : 0) + (size_t)g * D + c4, *vp = kv.v_pool + (vis ? at : 0) + (size_t)gv * E + c4;
      float* dst = st + (4 * j + kq) * (D + E) + c4;
#pragma unroll
      for (int i = 0; i < NI; i++) {
        if (32 * i < D) ar_copy16(dst + 32 * i, kp + 32 * i, vis ? 16 : 0);
        if (32 * i < E) ar_copy16(dst + D + 32 * i, vp + 32 * i, vis ? 16 : 0);
      }
    }
  };
  size_t row[AR_STAGES];
  unsigned late[AR_STAGES];                        // of the tile's eight keys those whose rows this step writes
#pragma unroll
  for (int i = 0; i < AR_STAGES; i++) row[i] = ti0 + i < ti_end ? row_of(ti0 + i) : (size_t)-1;
  if (early) {
    bool mine[AR_STAGES] = {};
    for (int r0 = 0; r0 < rows.n_rows; r0 += 32) {
      const int o = min(r0 + lane, rows.n_rows - 1);
      const size_t written = hyb_kv_row(kv, rows.seq_slot[rows.row_seq[o]], rows.pos[o], a.cache_layer);
      for (int j = 0; j < min(32, rows.n_rows - r0); j++) {
        const size_t w = __shfl_sync(THA_FULL_MASK, written, j);
#pragma unroll
        for (int i = 0; i < AR_STAGES; i++) mine[i] |= w == row[i];
      }
    }
#pragma unroll
    for (int i = 0; i < AR_STAGES; i++) late[i] = __ballot_sync(THA_FULL_MASK, mine[i]) & 0xFFu;
  } else {
#pragma unroll
    for (int i = 0; i < AR_STAGES; i++) late[i] = 0u;
  }
#pragma unroll
  for (int i = 0; i < AR_STAGES; i++)
    if (ti0 + i < ti_end) fetch(ti0 + i, row[i], ~late[i]);
  if (early) {
    pdl_wait();
#pragma unroll
    for (int i = 0; i < AR_STAGES; i++)
      if (late[i]) fetch(ti0 + i, row[i], late[i]);
  }
  ar_commit();
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
  for (int ti = ti0; ti < ti_end; ti++) {
    const int kt = tile_key(ti);
    float bias[GS][2];                                     // the distance's bias: asked for ahead of the tile, all at once
    if (a.rel) {
#pragma unroll
      for (int h = 0; h < GS; h++)
#pragma unroll
        for (int j = 0; j < 2; j++) bias[h][j] = hyb_attn_rel(a, g * gsize + min(h0 + h, gsize - 1), max(p - (kt + 4 * j + kq), 0));
    }
    if (ti == ti0) ar_await<0>();                          // the first round of the ring is one group, then a group a tile
    else if (ti >= ti0 + AR_STAGES) ar_await<AR_STAGES - 1>();
    __syncwarp();
    const float* st = ring + (size_t)((ti - ti0) % AR_STAGES) * 8 * (D + E);
    float s[GS][2];                                        // the scores of all heads, then their sums: nothing of one waits for another
    bool vis[2];
#pragma unroll
    for (int j = 0; j < 2; j++) {
      const int key = kt + 4 * j + kq;
      vis[j] = key <= p && key >= first && hyb_attn_sees(a, key, p, first);
      const float* src = st + (4 * j + kq) * (D + E) + c4;
      float4 kr[NI];
#pragma unroll
      for (int i = 0; i < NI; i++) kr[i] = 32 * i < D ? *reinterpret_cast<const float4*>(src + 32 * i) : make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
      for (int h = 0; h < GS; h++) {
        float d = 0.f;
#pragma unroll
        for (int i = 0; i < NI; i++) d = dot4(qv[h][i], kr[i], d);
        d += __shfl_xor_sync(THA_FULL_MASK, d, 1);
        d += __shfl_xor_sync(THA_FULL_MASK, d, 2);
        d += __shfl_xor_sync(THA_FULL_MASK, d, 4);
        d = d * a.scale * hs[h];
        if (a.softcap > 0.f) d = hyb_softcap(d, a.softcap);
        if (a.rel) d += bias[h][j];
        s[h][j] = vis[j] ? d : -INFINITY;
      }
    }
    float corr[GS];
#pragma unroll
    for (int h = 0; h < GS; h++) {
      const float m_new = fmaxf(m_run[h], fmaxf(s[h][0], s[h][1]));
      const bool any = m_new > -INFINITY;                  // else nothing was seen so far, and what there is stays
      corr[h] = any ? expf(m_run[h] - m_new) : 1.f;
      s[h][0] = any ? expf(s[h][0] - m_new) : 0.f;
      s[h][1] = any ? expf(s[h][1] - m_new) : 0.f;
      l_run[h] = l_run[h] * corr[h] + (s[h][0] + s[h][1]);
      m_run[h] = m_new;
    }
    const float *v0 = st + kq * (D + E) + D + c4, *v1 = v0 + 4 * (D + E);
#pragma unroll
    for (int i = 0; i < NI; i++) {
      const float4 x = 32 * i < E ? *reinterpret_cast<const float4*>(v0 + 32 * i) : make_float4(0.f, 0.f, 0.f, 0.f);
      const float4 y = 32 * i < E ? *reinterpret_cast<const float4*>(v1 + 32 * i) : make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
      for (int h = 0; h < GS; h++) {
        acc[h][i].x = fmaf(s[h][1], y.x, fmaf(s[h][0], x.x, acc[h][i].x * corr[h]));
        acc[h][i].y = fmaf(s[h][1], y.y, fmaf(s[h][0], x.y, acc[h][i].y * corr[h]));
        acc[h][i].z = fmaf(s[h][1], y.z, fmaf(s[h][0], x.z, acc[h][i].z * corr[h]));
        acc[h][i].w = fmaf(s[h][1], y.w, fmaf(s[h][0], x.w, acc[h][i].w * corr[h]));
      }
    }
    __syncwarp();
    if (ti + AR_STAGES < ti_end) fetch(ti + AR_STAGES, row_of(ti + AR_STAGES), ~0u);
    ar_commit();
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
template <typename T, int GS>
static int row_launch_heads(cudaStream_t s, const tha_attn_t* a, const tha_rows_t* rows, const tha_kv_t* kv, const float* q, T* out, int splits, float* partial,
                            const float* gate, long long ldg, int groups) {
  auto k = hyb_attn_row_kernel<T, GS>;
  const int ring = 4 * AR_STAGES * 8 * (a->dim + a->vdim) * (int)sizeof(float);
  THA_CUDA_OK(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, ring));
  THA_CUDA_OK(launch(k, dim3(rows->n_seqs * splits, a->kv_heads, groups), dim3(AR_THREADS), ring, s, pdl_enabled() != 0, *a, *rows, *kv, q, out, splits, partial,
                     gate, ldg, (int)(hyb_gemm_pdl() && rows->max_seq_rows == 1)));
  return THA_STATUS_SUCCESS;
}
template <typename T>
static int row_launch(cudaStream_t s, const tha_attn_t* a, const tha_rows_t* rows, const tha_kv_t* kv, const float* q, T* out, int splits, float* partial,
                      const float* gate, long long ldg) {
  const int gsize = a->heads / a->kv_heads, gs = gsize >= 3 ? AR_HEADS : gsize, groups = ceil_div(gsize, gs);
  if (gs == 1) return row_launch_heads<T, 1>(s, a, rows, kv, q, out, splits, partial, gate, ldg, groups);
  if (gs == 2) return row_launch_heads<T, 2>(s, a, rows, kv, q, out, splits, partial, gate, ldg, groups);
  return row_launch_heads<T, AR_HEADS>(s, a, rows, kv, q, out, splits, partial, gate, ldg, groups);
}
int hyb_attn_row_launch(cudaStream_t s, int dtype, const tha_attn_t* a, const tha_rows_t* rows, const tha_kv_t* kv, const float* q, void* out, int splits,
                        float* partial, const float* gate, long long ldg) {
  return dtype == THA_DT_BF16 ? row_launch(s, a, rows, kv, q, (__nv_bfloat16*)out, splits, partial, gate, ldg)
                              : row_launch(s, a, rows, kv, q, (float*)out, splits, partial, gate, ldg);
}
}  // namespace tha
