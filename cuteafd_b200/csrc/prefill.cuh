// What the two prompt attention kernels share: tile sizes, arguments, and the way from one to the other.
#pragma once

#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

namespace cafd {

constexpr int kHD = 128;          // head dim
constexpr int kBQ = 128;          // query rows of a tile
constexpr int kBKV = 128;         // kv tokens per tile (two 64-token pages)
constexpr int kPageTok = 64;
constexpr int kHalfBytes = 128 * 128;   // 128 rows x 64 bf16 (one swizzle atom wide) = 16 KiB
constexpr int kTileB = 2 * kHalfBytes;  // 32 KiB: a [128 x 128] bf16 tile as two 64-wide halves
constexpr int kPairSplits = 8;          // most shares of a row's keys
constexpr int kPairShareTiles = 8;      // least key tiles of a share (a row of fewer is cut into fewer shares)

struct PrefillDev {
  const int* page_table;   // [seqs, max_pages]
  const int* seq_lens;     // kv length per sequence (including this chunk)
  const int* q_start;      // [seqs + 1] row offsets into q/out
  __nv_bfloat16* out;      // [total_q, Hq, 128]
  uint32_t* status;
  int max_pages;
  int Hq, Hkv;
  int total_q;
  float scale_log2;
  int window;              // sliding window: a query at position t sees keys (t - window, t]; 0 = all earlier keys
  int keep;                // with a window: and the keys [0, keep)
  int ldo;                 // elements from row to row of out
  // kMaps == 2 only
  float lambda, out_scale, eps;
  // kMaps == 1 only
  const float* sink;              // [Hq] or null
  const __nv_bfloat16* gate;      // row t, head h: gate[t * gate_ld + h]; or null
  int gate_ld;
  const float2* v_table;          // [rows, 64] cos, sin; or null
  float cap_in, cap_log2;         // scale / cap, cap * log2(e); scale_log2 is then 1.  These two and v_table: kTurn only
  // kRope only
  const int* kv_tmp_start; // [seqs] first row of the sequence in the expansion buffers (multiple of 64)
  int q_head_stride;       // elements between heads in the nope query matrix (192 for [T, heads * 192])
  int qr_head_stride;      // elements between heads in the rope query matrix (576 for the absorbed-query buffer)
  int qr_col0;             // first rope column inside a head of that matrix (512)
};

// The two-tile kernel (attention_pair.cu).  maps: q, k, v, rope q, rope k.  splits > 1: `partial` holds splits * total_q * Hq * 130 floats.
int attn_pair(const CUtensorMap* maps, const PrefillDev& p, bool rope, int num_seqs, int max_q_len, float* partial, int splits, cudaStream_t st);

}  // namespace cafd
