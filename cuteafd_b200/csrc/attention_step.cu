// Attention of a plain decode step (one new token per sequence) in one launch: head norm, rotation and cache write of the new token, attention
// over the paged cache split over a cluster of blocks, and the merge of the splits through distributed shared memory.
//
// Bound: the cached keys and values, and at few rows the latencies of a chain of launches.  As kernels of their own the rotation, the attention
// (attention_decode.cu) and the merge of its partials each start behind their predecessor's end; here
//   * cached tokens older than this step are asked for before the programmatic-dependency wait, so that they travel under the projection whose
//     result the queries come from;
//   * every block norms and rotates its kv head's queries for itself (a few hundred cycles that the loads cover); the block that holds the last page
//     also makes the new key and value, stores them into the cache and puts them over the row that it loaded;
//   * a cluster is one (sequence, kv head): its blocks share the pages, leave O, maximum and sum in shared memory, and each merges its part of the
//     outputs from all of them in split order.
//
//   grid (sequence, kv head, split)   cluster (1, 1, splits)   block 128 threads (4 warps)
// The products are attention_decode.cu's: rows are the heads of the kv head (at most 16), a warp owns 16 of a page's 64 tokens, mma.sync m16n8k16.
#include <cooperative_groups.h>

#include "cafd_api.h"
#include "common.cuh"
#include "rope.cuh"

#include <atomic>

namespace cafd {

namespace cg = cooperative_groups;

constexpr int kSD = 128;
constexpr int kSPage = 64;
constexpr int kSTile = kSPage * kSD * 2;        // bytes of a page's keys (or values) of a kv head
constexpr int kStepMaxSplits = 16;

struct StepDev {
  const __nv_bfloat16* qkv;      // [T, (Hq + 2 Hkv) * 128]
  const __nv_bfloat16* q_norm;
  const __nv_bfloat16* k_norm;
  const __nv_bfloat16* bias;
  const float* inv_freq;
  const int* positions;
  const int* slots;
  __nv_bfloat16* k_cache;        // [pages, Hkv, 64, 128]
  __nv_bfloat16* v_cache;
  const int* page_table;
  const int* seq_lens;           // including the new token
  const int* q_start;
  __nv_bfloat16* out;            // rows of ldo elements
  int max_pages, Hq, Hkv, ldo, window, interleaved, rot, early;
  float eps, scale_log2;
};

__device__ __forceinline__ void step_cp16(uint32_t dst, const void* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
}
__device__ __forceinline__ void step_mma(float (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
               : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
               : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
__device__ __forceinline__ void step_ldmatrix_trans(uint32_t (&r)[4], const void* p) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(smem_u32(p)));
}

struct StepShared {
  float m[16], l[16];            // this block's share: maximum (log2 units) and sum of every row; its O (unnormalised) lies behind the warps' sums
  uint32_t q[16][kSD / 2 + 4];   // rotated queries, rows padded against bank conflicts
  uint32_t kv[2][kSD / 2];       // the new token's key and value
};

template <int kStages>
__global__ void __launch_bounds__(128) attn_step_kernel(const StepDev p) {
  extern __shared__ __align__(128) uint8_t smem[];          // ring of (keys, values) pages; the warps' sums at the end
  __shared__ StepShared sh;
  cg::cluster_group cluster = cg::this_cluster();
  const int seq = blockIdx.x, kvh = blockIdx.y, split = blockIdx.z, splits = gridDim.z;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, t4 = lane & 3;
  const int group = p.Hq / p.Hkv;

  if (!p.early) { pdl_wait(); pdl_trigger(); }
  const int row = p.q_start[seq];
  const bool live = p.q_start[seq + 1] > row;               // uniform over the cluster
  const int seq_len = live ? p.seq_lens[seq] : 0;
  const int lo = p.window > 0 ? max(0, seq_len - p.window) : 0;
  const int first_page = lo / kSPage, total_pages = (seq_len + kSPage - 1) / kSPage, n_pages = total_pages - first_page;
  const int per = (n_pages + splits - 1) / splits;
  const int p0 = first_page + min(n_pages, split * per), p1 = min(total_pages, p0 + per);
  const int* pt = p.page_table + static_cast<size_t>(seq) * p.max_pages;
  // 64 rows x 16 pieces of 16 bytes; the piece's place is XORed by the row so that fragment reads of 8 rows hit different banks
  auto load = [&](int pg) {
    const size_t at = (static_cast<size_t>(pt[pg]) * p.Hkv + kvh) * kSPage * kSD;
    const uint32_t d = smem_u32(smem) + ((pg - p0) % kStages) * 2 * kSTile;
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const int c = tid + i * 128, tok = c >> 4, ch = c & 15;
      const uint32_t to = d + tok * 256 + ((ch ^ (tok & 7)) << 4);
      step_cp16(to, p.k_cache + at + c * 8);
      step_cp16(to + kSTile, p.v_cache + at + c * 8);
    }
  };
  // (the new token's row of the last page is loaded as it stands, and replaced below)
#pragma unroll
  for (int s = 0; s < kStages - 1; ++s) {
    if (p0 + s < p1) load(p0 + s);
    asm volatile("cp.async.commit_group;" ::: "memory");
  }
  const bool own = live && p1 == total_pages && p0 < p1;    // this block holds the new token
  if (p.early) { pdl_wait(); pdl_trigger(); }
  if (live) {
    const int heads = p.Hq + 2 * p.Hkv;
    const HeadAngles ang = head_angles(static_cast<float>(p.positions[row]), p.inv_freq, lane, p.interleaved, p.rot);
    // items: the group's query heads, then the new key and value; rows past the group are zero
    for (int i = warp; i < group + (own ? 2 : 0); i += 4) {
      const int h = i < group ? kvh * group + i : i == group ? p.Hq + kvh : p.Hq + p.Hkv + kvh;
      const __nv_bfloat16* src = p.qkv + (static_cast<size_t>(row) * heads + h) * kSD;
      uint32_t a = *reinterpret_cast<const uint32_t*>(src + 2 * lane), b = *reinterpret_cast<const uint32_t*>(src + 64 + 2 * lane);
      if (p.bias) head_bias(a, b, p.bias + h * kSD, lane);
      if (i <= group) head_norm_rope(a, b, i < group ? p.q_norm : p.k_norm, p.eps, ang, lane, p.interleaved, p.rot);
      uint32_t* dst = i < group ? sh.q[i] : sh.kv[i - group];
      dst[lane] = a;
      dst[32 + lane] = b;
      const int slot = p.slots[row];
      if (i >= group && slot >= 0) {
        __nv_bfloat16* to = (i == group ? p.k_cache : p.v_cache) + ((static_cast<size_t>(slot >> 6) * p.Hkv + kvh) * kSPage + (slot & 63)) * kSD;
        *reinterpret_cast<uint32_t*>(to + 2 * lane) = a;
        *reinterpret_cast<uint32_t*>(to + 64 + 2 * lane) = b;
      }
    }
    for (int i = group * 64 + tid; i < 16 * 64; i += 128) sh.q[i >> 6][i & 63] = 0u;
  }
  __syncthreads();
  uint32_t qa[8][4];
#pragma unroll
  for (int ks = 0; ks < 8; ++ks)
#pragma unroll
    for (int half = 0; half < 2; ++half) {
      qa[ks][half] = live ? sh.q[g + 8 * half][8 * ks + t4] : 0u;
      qa[ks][half + 2] = live ? sh.q[g + 8 * half][8 * ks + 4 + t4] : 0u;
    }
  float m_run[2] = {-INFINITY, -INFINITY}, l_run[2] = {0.f, 0.f};
  float o_acc[16][4];
#pragma unroll
  for (int i = 0; i < 16; ++i) o_acc[i][0] = o_acc[i][1] = o_acc[i][2] = o_acc[i][3] = 0.f;

  for (int pg = p0; pg < p1; ++pg) {
    if (pg + kStages - 1 < p1) load(pg + kStages - 1);
    asm volatile("cp.async.commit_group;" ::: "memory");
    asm volatile("cp.async.wait_group %0;" ::"n"(kStages - 1) : "memory");
    __syncthreads();
    uint8_t* ks_ = smem + ((pg - p0) % kStages) * 2 * kSTile;
    const uint8_t* vs_ = ks_ + kSTile;
    if (own && pg == total_pages - 1) {
      const int tok = (seq_len - 1) & 63, ch = (tid & 63) >> 2;
      *reinterpret_cast<uint32_t*>(ks_ + (tid >> 6) * kSTile + tok * 256 + ((ch ^ (tok & 7)) << 4) + (tid & 3) * 4) = sh.kv[tid >> 6][tid & 63];
      __syncthreads();
    }
    // ---- S = Q K^T for this warp's 16 tokens
    float s[2][4];
#pragma unroll
    for (int nt = 0; nt < 2; ++nt) {
      s[nt][0] = s[nt][1] = s[nt][2] = s[nt][3] = 0.f;
      const int tok = warp * 16 + nt * 8 + g;
      const uint8_t* krow = ks_ + tok * 256;
#pragma unroll
      for (int ks = 0; ks < 8; ++ks) {
        const uint32_t b0 = *reinterpret_cast<const uint32_t*>(krow + (((2 * ks) ^ (tok & 7)) << 4) + 4 * t4);
        const uint32_t b1 = *reinterpret_cast<const uint32_t*>(krow + (((2 * ks + 1) ^ (tok & 7)) << 4) + 4 * t4);
        step_mma(s[nt], qa[ks], b0, b1);
      }
    }
    // ---- mask + online softmax (rows g and g + 8)
    const int tok0 = pg * kSPage + warp * 16;
    uint32_t pa[4];
    float corr[2];
#pragma unroll
    for (int half = 0; half < 2; ++half) {
      float mx = -INFINITY;
#pragma unroll
      for (int nt = 0; nt < 2; ++nt)
#pragma unroll
        for (int j = 0; j < 2; ++j) {
          const int tok = tok0 + nt * 8 + 2 * t4 + j;
          float& v = s[nt][2 * half + j];
          v = tok < seq_len && tok >= lo ? v * p.scale_log2 : -INFINITY;
          mx = fmaxf(mx, v);
        }
      mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 1));
      mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 2));
      const float m_new = fmaxf(m_run[half], mx), base = m_new == -INFINITY ? 0.f : m_new;
      corr[half] = m_new == -INFINITY ? 1.f : exp2f(m_run[half] - m_new);
      float rs = 0.f;
#pragma unroll
      for (int nt = 0; nt < 2; ++nt) {
        // rounded to bf16 first so that the row's sum matches what the product with V sees
        const uint32_t packed = pack_bf16(exp2f(s[nt][2 * half] - base), exp2f(s[nt][2 * half + 1] - base));
        rs += bf16_lo(packed) + bf16_hi(packed);
        pa[half + 2 * nt] = packed;
      }
      rs += __shfl_xor_sync(0xffffffffu, rs, 1);
      rs += __shfl_xor_sync(0xffffffffu, rs, 2);
      l_run[half] = l_run[half] * corr[half] + rs;
      m_run[half] = m_new;
    }
#pragma unroll
    for (int nd = 0; nd < 16; ++nd) {
      o_acc[nd][0] *= corr[0]; o_acc[nd][1] *= corr[0];
      o_acc[nd][2] *= corr[1]; o_acc[nd][3] *= corr[1];
    }
    // ---- O += P V
#pragma unroll
    for (int nd = 0; nd < 16; nd += 2) {
      const int m = lane >> 3, r = lane & 7, tok = warp * 16 + (m & 1) * 8 + r, ch = nd + (m >> 1);
      uint32_t vb[4];
      step_ldmatrix_trans(vb, vs_ + tok * 256 + ((ch ^ (tok & 7)) << 4));
      step_mma(o_acc[nd], pa, vb[0], vb[1]);
      step_mma(o_acc[nd + 1], pa, vb[2], vb[3]);
    }
    __syncthreads();
  }
  asm volatile("cp.async.wait_group 0;" ::: "memory");
  __syncthreads();

  // ---- the four warps, in order
  float* w_o = reinterpret_cast<float*>(smem);               // [4][16][128], then maxima and sums [4][16]
  float* w_m = w_o + 4 * 16 * kSD;
  float* w_l = w_m + 64;
  float* b_o = w_l + 64;                                     // [16][128]
#pragma unroll
  for (int nd = 0; nd < 16; ++nd) {
    float* o0 = w_o + (warp * 16 + g) * kSD + nd * 8 + 2 * t4;
    *reinterpret_cast<float2*>(o0) = make_float2(o_acc[nd][0], o_acc[nd][1]);
    *reinterpret_cast<float2*>(o0 + 8 * kSD) = make_float2(o_acc[nd][2], o_acc[nd][3]);
  }
  if (t4 == 0) {
    w_m[warp * 16 + g] = m_run[0]; w_m[warp * 16 + g + 8] = m_run[1];
    w_l[warp * 16 + g] = l_run[0]; w_l[warp * 16 + g + 8] = l_run[1];
  }
  __syncthreads();
  for (int r = 0; r < group; ++r) {                          // thread = value
    float M = -INFINITY, L = 0.f, O = 0.f;
#pragma unroll
    for (int w = 0; w < 4; ++w) M = fmaxf(M, w_m[w * 16 + r]);
#pragma unroll
    for (int w = 0; w < 4; ++w) {
      const float f = w_m[w * 16 + r] == -INFINITY ? 0.f : exp2f(w_m[w * 16 + r] - M);
      L += w_l[w * 16 + r] * f;
      O += w_o[(w * 16 + r) * kSD + tid] * f;
    }
    b_o[r * kSD + tid] = O;
    if (tid == 0) { sh.m[r] = M; sh.l[r] = L; }
  }
  // ---- the cluster's blocks, in order: this one takes every splits-th run of 32 values
  cluster.sync();
  for (int c = split * 4 + warp; live && c < group * 4; c += splits * 4) {
    const int r = c >> 2, d = (c & 3) * 32 + lane;
    float m[kStepMaxSplits], l[kStepMaxSplits], o[kStepMaxSplits], M = -INFINITY, L = 0.f, O = 0.f;
#pragma unroll
    for (int s = 0; s < kStepMaxSplits; ++s) {
      m[s] = -INFINITY; l[s] = o[s] = 0.f;
      if (s < splits) {
        const StepShared* from = cluster.map_shared_rank(&sh, s);
        m[s] = from->m[r]; l[s] = from->l[r]; o[s] = *cluster.map_shared_rank(b_o + r * kSD + d, s);
      }
    }
#pragma unroll
    for (int s = 0; s < kStepMaxSplits; ++s) M = fmaxf(M, m[s]);
#pragma unroll
    for (int s = 0; s < kStepMaxSplits; ++s) {
      const float f = m[s] == -INFINITY ? 0.f : exp2f(m[s] - M);
      L += l[s] * f;
      O += o[s] * f;
    }
    p.out[static_cast<size_t>(row) * p.ldo + (kvh * group + r) * kSD + d] = __float2bfloat16(L > 0.f ? O / L : 0.f);
  }
  cluster.sync();                                            // no block leaves while another reads its share
}

template <int kStages>
static int launch_step(const StepDev& p, int num_seqs, int splits, cudaStream_t st) {
  constexpr int kSmem = kStages * 2 * kSTile;
  static_assert(kSmem >= (5 * 16 * kSD + 128) * 4, "the warps' sums and the block's");
  auto kern = attn_step_kernel<kStages>;
  static std::atomic<unsigned long long> set{0};             // the attributes are the device's
  int dev = 0;
  CAFD_CHECK_CUDA(cudaGetDevice(&dev));
  const unsigned long long bit = 1ull << (dev & 63);
  if (dev > 63 || !(set.load(std::memory_order_relaxed) & bit)) {
    CAFD_CHECK_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmem));
    CAFD_CHECK_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeNonPortableClusterSizeAllowed, 1));
    set.fetch_or(bit, std::memory_order_relaxed);
  }
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(num_seqs, p.Hkv, splits);
  cfg.blockDim = dim3(128);
  cfg.dynamicSmemBytes = kSmem;
  cfg.stream = st;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = pdl_enabled() ? 1 : 0;
  attr[1].id = cudaLaunchAttributeClusterDimension;
  attr[1].val.clusterDim.x = attr[1].val.clusterDim.y = 1;
  attr[1].val.clusterDim.z = splits;
  cfg.attrs = attr;
  cfg.numAttrs = 2;
  CAFD_CHECK_CUDA(cudaLaunchKernelEx(&cfg, kern, p));
  return static_cast<int>(cudaGetLastError());
}

}  // namespace cafd

using namespace cafd;

// Blocks that share a (sequence, kv head) of a decode step, 1 to 16; 0 where the step is left to the rotation, the split attention and its merge:
// more heads to a kv head than a tile has rows, fixed splits, or so few rows of so long a context that sixteen blocks a kv head would leave SMs
// idle.  Some 320 blocks run at once; with many rows six of them, where each has pages enough, even out rows of different lengths.  Projections and
// attention of a layer of 32 / 4 heads in a graph, us, rotation, attention and merge apart / in one launch with 1 / 2 / 4 / 8 / 16 blocks:
//   1 row of 8192  31.6   104 / 62 / 40.5 / 29.7 / 25.0       8 rows of 8192       52.6   107 / 64.1 / 43.7 / 42.8 / 52.3 (10: 42.9)
//   1 row of 500   25.5   28.6 / 23.8 / 21.4 / 20.2           16 rows of 8192      95.5   111 / 69.2 / 67.4 / 80.5 / 91.6 (5: 64.5)
//   3 rows of 500  25.7   28.8 / 24.1 / 21.3 / 20.3           32 rows of 8192      152    127 / 121 / 148 / 141 / 173 (6: 126)
//   4 rows of 4000 34.4   64.6 / 42.3 / 30.9 / - / 27.2       32 of 2048 to 8192   117    129 / 116 / 109 / 110 / 136 (6: 103)
extern "C" int cafd_attn_step_splits(int num_seqs, int max_pages, int Hq, int Hkv, int window, int num_sms) {
  if (num_seqs < 1 || Hkv < 1 || Hq % Hkv || Hq / Hkv > 16 || max_pages < 1 || fixed_kv_split_tokens() > 0) return 0;
  const long long sms = num_sms > 0 ? num_sms : 148, tiles = static_cast<long long>(num_seqs) * Hkv;
  long long pages = max_pages;
  if (window > 0 && (window + kSPage - 1) / kSPage + 1 < pages) pages = (window + kSPage - 1) / kSPage + 1;
  const long long even = (pages + 21) / 22;
  long long s = 320 * sms / 148 / tiles;
  if (s < 4) s = s > even ? s : even < 6 ? even : 6;
  if (s > pages) s = pages;
  if (s > kStepMaxSplits) s = kStepMaxSplits;
  if (s < 1) s = 1;
  return pages > 16 * s && tiles * s < sms ? 0 : static_cast<int>(s);
}

// qkv [T, (Hq + 2 Hkv) * 128] of one token per sequence (q_start: at most one row each); the new keys and values go to their slots of the caches
// (negative: nowhere), out row t, head h: out[t * ldo + 128 h].  q_norm / k_norm / bias may be null; rot 128 or 64 rotated dims.  early: tables,
// lengths and the cached tokens before this step's are not written by the previous kernel of the stream.
extern "C" int cafd_attn_step(const void* qkv, const void* q_norm, const void* k_norm, const void* bias, const float* inv_freq, const int* positions,
                              const int* slots, void* k_cache, void* v_cache, const int* page_table, const int* seq_lens, const int* q_start,
                              void* out, int ldo, int num_seqs, int max_pages, int Hq, int Hkv, int D, int rot, int interleaved, float eps,
                              float scale, int window, int splits, int early, cafd_stream_t s) {
  if (num_seqs <= 0) return 0;
  if (D != kSD || Hkv < 1 || Hq % Hkv || Hq / Hkv > 16 || (rot != 128 && rot != 64) || window < 0 || ldo < Hq * kSD || max_pages < 1) return -10;
  if (splits < 1 || splits > kStepMaxSplits || !slots || !positions || !inv_freq) return -10;
  StepDev p{};
  p.qkv = static_cast<const __nv_bfloat16*>(qkv);
  p.q_norm = static_cast<const __nv_bfloat16*>(q_norm); p.k_norm = static_cast<const __nv_bfloat16*>(k_norm);
  p.bias = static_cast<const __nv_bfloat16*>(bias);
  p.inv_freq = inv_freq; p.positions = positions; p.slots = slots;
  p.k_cache = static_cast<__nv_bfloat16*>(k_cache); p.v_cache = static_cast<__nv_bfloat16*>(v_cache);
  p.page_table = page_table; p.seq_lens = seq_lens; p.q_start = q_start;
  p.out = static_cast<__nv_bfloat16*>(out);
  p.max_pages = max_pages; p.Hq = Hq; p.Hkv = Hkv; p.ldo = ldo; p.window = window; p.interleaved = interleaved; p.rot = rot; p.early = early;
  p.eps = eps; p.scale_log2 = scale * 1.4426950408889634f;
  int dev = 0, sms = 148;
  CAFD_CHECK_CUDA(cudaGetDevice(&dev));
  CAFD_CHECK_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
  cudaStream_t st = static_cast<cudaStream_t>(s);
  // Four pages in flight where a block has an SM to itself.  A cluster needs its SMs within one GPC, so that 128 such blocks in clusters of eight don't
  // run at once (4 rows of 4000 tokens in eight: 36.8 us, 31.0 with two pages in flight); 96 do (3 rows of 500 in eight: 20.3 us, 22.5).
  const long long blocks = static_cast<long long>(num_seqs) * Hkv * splits;
  return blocks <= (splits <= 4 ? sms : sms * 2 / 3) ? launch_step<4>(p, num_seqs, splits, st) : launch_step<2>(p, num_seqs, splits, st);
}
