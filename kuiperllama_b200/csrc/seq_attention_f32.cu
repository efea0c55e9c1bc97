// Prompt attention of the sequence-batch engine in fp32: the problem of attention_mma_kernel (seq_attention_mma.cu) -- a CTA takes
// 64 consecutive rows of one entry and one key/value head, row r = token r / rep, query head g * rep + r % rep -- on fp32
// multiply-adds, by the loop of f32_attention.cuh.  With one split the kernel divides by the sum, joins the sink and applies the
// output gate itself; with several it leaves (max, sum, unnormalised output) per split for attention_merge_kernel.
//
// The split-key kernel that these steps took before (attention_kernel, 32 rows against 64 keys) brings keys in by scalar loads
// between two barriers and reads two 4-byte operands from shared memory for every four multiply-adds of a score; it stays for few
// rows and for head sizes past 128.
#include <cuda_runtime.h>

#include <cstdint>

#include "f32_attention.cuh"
#include "seq_engine.h"
#include "seq_mma.cuh"

namespace kllm {
namespace seq {
namespace {

struct PagedWork {
  const AttnShape& a;
  const float *qb, *kb, *vb;
  const int32_t* table;
  const PagedKV& kv;
  int r0, n_rows, first, pos0, rep, g, gv, pmax;
  int keep_tiles, tile_first, tile_lo, n_tiles;
  int pos_lo, seen_hi;  // the first row's position, the first key that the last row sees

  __device__ __forceinline__ bool keys_by_chunk() const { return false; }
  __device__ __forceinline__ const float* any() const { return kb; }
  __device__ __forceinline__ const float* q(int row) const {
    const int r = r0 + row;
    return r < n_rows ? qb + (static_cast<size_t>(first + r / rep) * a.heads + g * rep + r % rep) * a.dim : nullptr;
  }
  __device__ __forceinline__ size_t slot(int j) const { return static_cast<size_t>(table[j / kv.page]) * kv.page + j % kv.page; }
  __device__ __forceinline__ const float* key(int j, int c) const {
    return j <= pmax ? kb + slot(j) * kv.k_row + g * a.dim + c * 4 : nullptr;
  }
  __device__ __forceinline__ const float* value(int j, int c) const {
    return j <= pmax ? vb + slot(j) * kv.v_row + gv * a.vdim + c * 4 : nullptr;
  }
  __device__ __forceinline__ int tile(int i) const {
    const int li = tile_lo + i;
    return li < keep_tiles ? li : tile_first + (li - keep_tiles);
  }
  __device__ __forceinline__ bool hidden(int row, int j) const {
    const int r = r0 + row;
    const int p = pos0 + r / rep;
    return r >= n_rows || j > p || (j < first_seen(a, p) && j >= a.keep_first);
  }
  __device__ __forceinline__ bool whole(int t) const {
    return r0 + f32attn::kRows <= n_rows && t * f32attn::kKeys + f32attn::kKeys - 1 <= pos_lo && t * f32attn::kKeys >= seen_hi;
  }
  __device__ __forceinline__ float score(float s) const {
    s *= a.scale;
    return a.softcap > 0.f ? a.softcap * tanhf(s / a.softcap) : s;
  }
};

template <int NV>
__global__ void __launch_bounds__(f32attn::kThreads)
attention_f32_kernel(AttnShape a, const float* __restrict__ q, PagedKV kv, const int32_t* __restrict__ ent_first,
                     const int32_t* __restrict__ ent_count, const int32_t* __restrict__ ent_seq,
                     const int32_t* __restrict__ ent_pos0, int splits, float* __restrict__ ws, const float* __restrict__ gates,
                     float* __restrict__ out) {
  extern __shared__ __align__(16) float sm[];
  const int e = blockIdx.x / a.kv_heads, g = blockIdx.x % a.kv_heads, split = blockIdx.z;
  const int rep = a.heads / a.kv_heads;
  const int first = ent_first[e], pos0 = ent_pos0[e], n_rows = ent_count[e] * rep;
  const int r0 = (gridDim.y - 1 - blockIdx.y) * f32attn::kRows;  // the tiles with the most keys start first
  if (r0 >= n_rows) return;
  const int last_row = min(r0 + f32attn::kRows, n_rows) - 1;
  const int pmax = pos0 + last_row / rep;  // last position any row of the tile sees
  const int n_tiles = pmax / f32attn::kKeys + 1;
  // with a window or chunks no row of the tile sees anything before what its first row sees; tiles before that which hold kept
  // first positions come ahead: this CTA's list of tiles is [0, keep_tiles) then [tile_first, n_tiles), cut into `splits` parts
  const int tile_first = first_seen(a, pos0 + r0 / rep) / f32attn::kKeys;
  const int keep_tiles = min(tile_first, (a.keep_first + f32attn::kKeys - 1) / f32attn::kKeys);
  const int list_n = keep_tiles + n_tiles - tile_first, per = (list_n + splits - 1) / splits;
  const int tile_lo = split * per, tile_hi = min(list_n, tile_lo + per);
  const PagedWork w{a, q, static_cast<const float*>(kv.k), static_cast<const float*>(kv.v),
                    kv.table + static_cast<size_t>(ent_seq[e]) * kv.table_stride, kv, r0, n_rows, first, pos0, rep, g,
                    g / v_share_of(a), pmax, keep_tiles, tile_first, tile_lo, max(0, tile_hi - tile_lo), pos0 + r0 / rep,
                    first_seen(a, pmax)};
  f32attn::Sums<NV> r;
  f32attn::attend<NV>(w, a.dim, a.vdim, sm, r);

  const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4, vdim = a.vdim;
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int rr = r0 + ty + 16 * i;
    if (rr >= n_rows) continue;
    const size_t th = static_cast<size_t>(first + rr / rep) * a.heads + g * rep + rr % rep;
    if (splits == 1 && !a.no_merge) {
      float l = r.l[i];
      if (a.sink != nullptr)  // exp(sink) joins the denominator
        l = r.m[i] > -INFINITY ? l + expf(a.sink[th % a.heads] - r.m[i]) : 1.0f;
      const bool per_element = gates != nullptr && a.gate == KLLM_SEQ_GATE_ELEMENT;
      const float head_gate = gates && !per_element ? gates[th] : 1.0f;
#pragma unroll
      for (int n = 0; n < NV; ++n) {
        const int col = n * 64 + tx * 4;
        if (col >= vdim) break;
        float4 gt = make_float4(head_gate, head_gate, head_gate, head_gate);
        if (per_element) {
          const float* ge = gates + th * vdim + col;
          gt = make_float4(ge[0], ge[1], ge[2], ge[3]);
        }
        *reinterpret_cast<float4*>(out + th * vdim + col) =
            make_float4(r.o[i][n * 4] / l * gt.x, r.o[i][n * 4 + 1] / l * gt.y, r.o[i][n * 4 + 2] / l * gt.z,
                        r.o[i][n * 4 + 3] / l * gt.w);
      }
    } else {
      float* p = ws + (th * splits + split) * (vdim + 2);
      if (tx == 0) p[0] = r.m[i], p[1] = r.l[i];
#pragma unroll
      for (int n = 0; n < NV; ++n)
#pragma unroll
        for (int c = 0; c < 4; ++c)
          if (n * 64 + tx * 4 + c < vdim) p[2 + n * 64 + tx * 4 + c] = r.o[i][n * 4 + c];
    }
  }
}

}  // namespace

// Steps with enough rows per key head to fill tiles of 64; heads whose keys and values are whole 16-byte chunks.
bool attention_f32_usable(int dtype, const AttnShape& a, const PagedKV& kv, int max_count) {
  static const bool off = [] { const char* e = getenv("KLLM_SEQ_F32_TILES"); return e != nullptr && e[0] == '0'; }();
  if (off || dtype != KLLM_SEQ_F32 || a.kv_heads <= 0 || a.heads % a.kv_heads || kv.table == nullptr) return false;
  const bool dims = a.dim % 4 == 0 && a.dim <= 128 && a.vdim % 4 == 0 && a.vdim <= 128 && kv.k_row % 4 == 0 && kv.v_row % 4 == 0;
  return dims && max_count >= 2 && max_count * (a.heads / a.kv_heads) >= 16;
}

template <int NV>
static int launch_f32(const AttnShape& a, const void* q, const float* gates, const PagedKV& kv, int n_entries,
                      const int32_t* ent_first, const int32_t* ent_count, const int32_t* ent_seq, const int32_t* ent_pos0,
                      int max_count, int splits, float* ws, void* out, cudaStream_t s) {
  const cudaError_t e = cudaFuncSetAttribute(attention_f32_kernel<NV>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                             static_cast<int>(f32attn::smem_floats(128, NV) * sizeof(float)));
  if (e != cudaSuccess) return cuda_rc(e);
  const int rep = a.heads / a.kv_heads;
  const dim3 grid(n_entries * a.kv_heads, (max_count * rep + f32attn::kRows - 1) / f32attn::kRows, splits);
  if (grid.y > 65535u) return KLLM_E_UNSUPPORTED;
  attention_f32_kernel<NV><<<grid, f32attn::kThreads, f32attn::smem_floats(a.dim, NV) * sizeof(float), s>>>(
      a, static_cast<const float*>(q), kv, ent_first, ent_count, ent_seq, ent_pos0, splits, ws, a.gate ? gates : nullptr,
      static_cast<float*>(out));
  count_launch();
  return cuda_rc(cudaGetLastError());
}

int launch_attention_f32(const AttnShape& a, const void* q, const float* gates, const PagedKV& kv, int n_entries,
                         const int32_t* ent_first, const int32_t* ent_count, const int32_t* ent_seq, const int32_t* ent_pos0,
                         int max_count, int splits, float* ws, void* out, cudaStream_t s) {
  if (a.vdim <= 64)
    return launch_f32<1>(a, q, gates, kv, n_entries, ent_first, ent_count, ent_seq, ent_pos0, max_count, splits, ws, out, s);
  return launch_f32<2>(a, q, gates, kv, n_entries, ent_first, ent_count, ent_seq, ent_pos0, max_count, splits, ws, out, s);
}

}  // namespace seq
}  // namespace kllm
