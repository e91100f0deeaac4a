// Causal prompt attention over the paged KV cache, two query tiles to a block (head_dim 128).
//
// Bound: per tile of 128 queries x 128 keys the tensor core works 1024 cycles (S = Q K^T and O += P V) and the special-function unit as long on
// 16384 exponentials; either waits for the other's result.  So a block holds two tiles that don't: while one tile's scores turn into weights
// on four softmax warps, the other's products run.  The two share every key and value tile: they are two query heads of one kv head (GQA), or
// two neighbouring row tiles of one head (kRope, expanded MLA, where every head has keys of its own).
//
//   warp 0     TMA producer: both Q tiles once, then K and V tiles in rings of their own
//   warp 1     MMA issuer: per tile and key tile P V, then at once the next Q K^T of the same query tile
//   warps 4-7, 8-11  softmax of query tile 0, 1: thread = row.  A row of 128 scores goes to registers with one wait, becomes P as bf16 pairs over
//              the columns its scores came from (the A operand of P V is read from tensor memory), and O is rescaled only when the reference
//              maximum moved (a row maximum exceeds it by more than 8 in log2 units).
// TMEM: S of the two tiles (128 columns each, P over the first 64), O of the two (128 each).  A score buffer needs no barrier of its own: Q K^T is
// issued behind the P V that reads P, so it overwrites scores and weights that have been read; and scores that are there mean that every earlier
// P V has ended, so O may be rescaled.
//
// Measured against one tile per block (attention_prefill.cu), 32 / 4 heads: 8192 rows 707 -> 463 us (1188 TFLOP/s, 0.83 of the sustained rate; with
// the exponentials left out 417), 4096 214 -> 132, 2048 75 -> 43, 512 behind 16384 184 -> 149.  Left out, as slower: the first half of the next
// scores issued before P stands (507), P handed over in halves (474), every fourth or second exponential as a polynomial (465, 494).
//
// Keys split over blocks (splits > 1, where a step has fewer block pairs than the chip has SMs): a block takes a share of the key tiles and leaves
// O, maximum and sum as fp32; attn_pair_merge_kernel adds the shares in order.
#include "cafd_api.h"
#include "common.cuh"
#include "host_tma.h"
#include "prefill.cuh"

#include <atomic>

namespace cafd {

constexpr int kPairThreads = 384;
// Registers per thread: launched with 168 (three warpgroups, 504 in all); a softmax thread holds a row of 128 scores.
constexpr int kPairRegsControl = 56, kPairRegsSoftmax = 224;
static_assert(kPairRegsControl + 2 * kPairRegsSoftmax <= 168 * 3, "the launch's registers");
constexpr int kPairStat = 2;                       // floats beside a partial row: maximum, sum

template <bool kRope>
struct PairCfg {
  static constexpr int kKS = kRope ? 2 : 3, kVS = kRope ? 1 : 2;              // stages
  static constexpr int kQBytes = kTileB + (kRope ? kHalfBytes : 0);          // of one query tile
  static constexpr int kKBytes = kTileB + (kRope ? kHalfBytes : 0);
  static constexpr int kSmem = 2 * kQBytes + kKS * kKBytes + kVS * kTileB + 1024;
  static_assert(kSmem <= 227 * 1024 - 512, "shared memory");
};

__device__ __forceinline__ uint64_t pair_f32x2(float a, float b) {
  uint64_t r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
  return r;
}

template <bool kRope>
__global__ void __launch_bounds__(kPairThreads, 1)
attn_pair_kernel(const __grid_constant__ CUtensorMap tm_q, const __grid_constant__ CUtensorMap tm_k, const __grid_constant__ CUtensorMap tm_v,
                 const __grid_constant__ CUtensorMap tm_qr, const __grid_constant__ CUtensorMap tm_kr, const PrefillDev p, float* partial,
                 int splits) {
  using Cfg = PairCfg<kRope>;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* sQ = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));      // a tile: 128 x 128 (+ 128 x 64)
  uint8_t* sK = sQ + 2 * Cfg::kQBytes;
  uint8_t* sV = sK + Cfg::kKS * Cfg::kKBytes;
  __shared__ uint64_t q_full, k_full[Cfg::kKS], k_empty[Cfg::kKS], v_full[Cfg::kVS], v_empty[Cfg::kVS], s_full[2], p_ready[2], o_full[2];
  __shared__ uint32_t tmem_slot;

  pdl_wait();
  pdl_trigger();
  const int warp = warp_uniform(threadIdx.x >> 5), lane = threadIdx.x & 31;
  const int seq = blockIdx.z / splits, split = blockIdx.z - seq * splits;
  const int head0 = kRope ? blockIdx.x : 2 * blockIdx.x;
  const int kvh = head0 / (p.Hq / p.Hkv);
  const int q0 = p.q_start[seq];
  const int q_len = p.q_start[seq + 1] - q0;
  const int kv_len = p.seq_lens[seq];
  constexpr int kRowsPerBlock = kRope ? 2 * kBQ : kBQ;
  const int bt = (q_len + kRowsPerBlock - 1) / kRowsPerBlock - 1 - static_cast<int>(blockIdx.y);      // heaviest blocks first
  if (bt < 0) return;
  const int row0 = bt * kRowsPerBlock;                               // first query row of the block (within the chunk)
  const int pos0 = kv_len - q_len + row0;                            // its absolute position
  // key tiles in the order that they are walked: with a sliding window the kept first ones, then the window's; tile of ordinal j is
  // j + (j < kept_tiles ? 0 : tile0)
  const int win_tile = p.window > 0 ? max(0, pos0 - p.window + 1) / kBKV : 0;
  const int kept_tiles = p.window > 0 ? min((p.keep + kBKV - 1) / kBKV, win_tile) : 0;
  const int tile0 = win_tile - kept_tiles;
  auto tiles_of = [&](int rows0) { return rows0 < q_len ? min(kv_len - q_len + rows0 + kBQ - 1, kv_len - 1) / kBKV + 1 - tile0 : 0; };
  const int all0 = tiles_of(row0), all1 = kRope ? tiles_of(row0 + kBQ) : all0;       // (kRope: the second tile has more, or no rows at all)
  const int all = max(all0, all1);
  const int shares = max(1, min(splits, all / kPairShareTiles));
  const int jb = split < shares ? split * all / shares : all, je = split < shares ? (split + 1) * all / shares : all;      // this block's share
  const int n0 = max(0, min(all0, je) - jb), n1 = max(0, min(all1, je) - jb), n = je - jb;
  const int seq_pages = (kv_len + kPageTok - 1) / kPageTok;

  if (threadIdx.x == 0) {
    mbar_init(&q_full, 1);
    for (int i = 0; i < Cfg::kKS; ++i) { mbar_init(&k_full[i], 1); mbar_init(&k_empty[i], 1); }
    for (int i = 0; i < Cfg::kVS; ++i) { mbar_init(&v_full[i], 1); mbar_init(&v_empty[i], 1); }
    for (int i = 0; i < 2; ++i) { mbar_init(&s_full[i], 1); mbar_init(&p_ready[i], 4); mbar_init(&o_full[i], 1); }
    mbar_fence_init();
  }
  if (warp == 1) {
    tmem_alloc(&tmem_slot, 512);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = tmem_slot;               // S at 128 i, O at 256 + 128 i

  if (warp < 4) reg_dec<kPairRegsControl>();

  if (warp == 0) {
    if (lane == 0 && n > 0) {
      tma_prefetch_desc(&tm_q); tma_prefetch_desc(&tm_k); tma_prefetch_desc(&tm_v);
      if (kRope) { tma_prefetch_desc(&tm_qr); tma_prefetch_desc(&tm_kr); }
      const int two = !kRope || all1 > 0;
      mbar_expect_tx(&q_full, (1 + two) * Cfg::kQBytes);
      for (int i = 0; i <= two; ++i) {
        uint8_t* d = sQ + i * Cfg::kQBytes;
        const int col = kRope ? head0 * p.q_head_stride : (head0 + i) * kHD, r = q0 + row0 + (kRope ? i * kBQ : 0);
        tma_load_2d(d, &tm_q, &q_full, col, r);
        tma_load_2d(d + kHalfBytes, &tm_q, &q_full, col + 64, r);
        if (kRope) tma_load_2d(d + kTileB, &tm_qr, &q_full, head0 * p.qr_head_stride + p.qr_col0, r);
      }
      const int* pt = p.page_table + static_cast<size_t>(seq) * p.max_pages;
      const int tmp_page0 = kRope ? p.kv_tmp_start[seq] / kPageTok : 0;
      auto page = [&](int pg) { return pg < seq_pages ? pt[pg] : 0; };           // page 0 is the all-zero page
      bool ok = true;
      for (int j = 0; ok && j < n; ++j) {
        const int t = jb + j, pg = 2 * (t + (t < kept_tiles ? 0 : tile0));
        const int pa = page(pg), pb = page(pg + 1);
        // expanded K / V (kRope) sit in order in their buffer: "page" = row block of 64; past the end TMA fills zeros
        const int ka = kRope ? tmp_page0 + pg : pa, kb = kRope ? tmp_page0 + pg + 1 : pb;
        const int ks = j % Cfg::kKS, vs = j % Cfg::kVS;
        if (!mbar_wait(&k_empty[ks], ((j / Cfg::kKS) & 1) ^ 1, p.status, kTimeoutEmptyBarrier)) break;
        uint8_t* kd = sK + ks * Cfg::kKBytes;
        mbar_expect_tx(&k_full[ks], Cfg::kKBytes);
        tma_load_4d(kd, &tm_k, &k_full[ks], 0, kvh, 0, ka);
        tma_load_4d(kd + 64 * 128, &tm_k, &k_full[ks], 0, kvh, 0, kb);
        tma_load_4d(kd + kHalfBytes, &tm_k, &k_full[ks], 64, kvh, 0, ka);
        tma_load_4d(kd + kHalfBytes + 64 * 128, &tm_k, &k_full[ks], 64, kvh, 0, kb);
        if (kRope) {
          tma_load_3d(kd + kTileB, &tm_kr, &k_full[ks], 512, 0, pa);
          tma_load_3d(kd + kTileB + 64 * 128, &tm_kr, &k_full[ks], 512, 0, pb);
        }
        if (!mbar_wait(&v_empty[vs], ((j / Cfg::kVS) & 1) ^ 1, p.status, kTimeoutEmptyBarrier)) break;
        uint8_t* vd = sV + vs * kTileB;
        mbar_expect_tx(&v_full[vs], kTileB);
        tma_load_4d(vd, &tm_v, &v_full[vs], 0, kvh, 0, ka);
        tma_load_4d(vd + 64 * 128, &tm_v, &v_full[vs], 0, kvh, 0, kb);
        tma_load_4d(vd + kHalfBytes, &tm_v, &v_full[vs], 64, kvh, 0, ka);
        tma_load_4d(vd + kHalfBytes + 64 * 128, &tm_v, &v_full[vs], 64, kvh, 0, kb);
      }
    }
  } else if (warp == 1) {
    if (n > 0) {
      constexpr uint32_t idesc_qk = make_idesc(128, 128, 1, 1, 0, 0);
      constexpr uint32_t idesc_pv = make_idesc(128, 128, 1, 1, 0, 1);   // B = V is MN-major
      const uint64_t dQ = smem_desc_k_sw128(smem_u32(sQ)), dK = smem_desc_k_sw128(smem_u32(sK));
      const uint64_t dV = smem_desc_mn_sw128(smem_u32(sV), kHalfBytes);
      auto last = [&](int i, int j) { return i == 1 || j >= n1; };      // no other tile reads key tile j after query tile i
      auto issue_qk = [&](int i, int j) -> bool {
        const int st = j % Cfg::kKS;
        if (!mbar_wait_warp(&k_full[st], (j / Cfg::kKS) & 1, p.status, kTimeoutFullBarrier)) return false;
        tc_fence_after();
        if (elect_one()) {
          const uint64_t a = dQ + static_cast<uint64_t>(i * (Cfg::kQBytes >> 4)), b = dK + static_cast<uint64_t>(st * (Cfg::kKBytes >> 4));
#pragma unroll
          for (int k = 0; k < (kRope ? 12 : 8); ++k)
            umma_f16(tmem + i * 128, a + (k >> 2) * (kHalfBytes >> 4) + (k & 3) * 2, b + (k >> 2) * (kHalfBytes >> 4) + (k & 3) * 2, idesc_qk, k ? 1u : 0u);
          umma_commit(&s_full[i]);
          if (last(i, j)) umma_commit(&k_empty[st]);
        }
        __syncwarp();
        return true;
      };
      bool ok = mbar_wait_warp(&q_full, 0, p.status, kTimeoutFullBarrier);
      if (n0 > 0) ok = ok && issue_qk(0, 0);
      if (n1 > 0) ok = ok && issue_qk(1, 0);
      for (int j = 0; ok && j < n; ++j) {
        const int vs = j % Cfg::kVS;
#pragma unroll
        for (int i = 0; i < 2; ++i) {
          const int ni = i ? n1 : n0;
          if (!ok || j >= ni) continue;
          ok = mbar_wait_warp(&v_full[vs], (j / Cfg::kVS) & 1, p.status, kTimeoutFullBarrier) &&
               mbar_wait_warp(&p_ready[i], j & 1, p.status, kTimeoutSoftmax);
          if (!ok) continue;
          tc_fence_after();
          if (elect_one()) {
            const uint64_t b = dV + static_cast<uint64_t>(vs * (kTileB >> 4));
#pragma unroll
            for (int k8 = 0; k8 < 8; ++k8)      // B: 16 kv rows per step (2 KiB), two 64-wide d halves 16 KiB apart
              umma_f16_ts(tmem + 256 + i * 128, tmem + i * 128 + k8 * 8, b + (k8 * 2048 >> 4), idesc_pv, (j | k8) ? 1u : 0u);
            if (last(i, j)) umma_commit(&v_empty[vs]);
            if (j == ni - 1) umma_commit(&o_full[i]);
          }
          __syncwarp();
          if (j + 1 < ni) ok = issue_qk(i, j + 1);
        }
      }
    }
  } else if (warp >= 4) {
    reg_inc<kPairRegsSoftmax>();
    const int i = warp >= 8, quad = warp & 3;
    const int row = quad * 32 + lane;                // row within the tile = TMEM lane
    const int rows0 = row0 + (kRope ? i * kBQ : 0), head = kRope ? head0 : head0 + i;
    const int tpos0 = pos0 + (kRope ? i * kBQ : 0), rowpos = tpos0 + row;
    const uint32_t tS = tmem + i * 128 + (static_cast<uint32_t>(quad * 32) << 16), tO = tS + 256;
    const int ni = i ? n1 : n0;
    float m_run = -INFINITY, l_half[2] = {0.f, 0.f};        // sums of the tiles' two column halves, as the one-tile kernel keeps them
    const uint64_t scale2 = pair_f32x2(p.scale_log2, p.scale_log2);
    bool ok = true;
    for (int j = 0; j < ni; ++j) {
      if (!mbar_wait_warp(&s_full[i], j & 1, p.status, kTimeoutTmemFull)) { ok = false; break; }
      tc_fence_after();
      const int t = jb + j, col0 = (t + (t < kept_tiles ? 0 : tile0)) * kBKV;        // first kv position of this tile
      uint32_t r[128];
#pragma unroll
      for (int c = 0; c < 4; ++c) tmem_ld_32x32(tS + c * 32, *reinterpret_cast<uint32_t(*)[32]>(r + c * 32));
      tmem_ld_wait();
      // uniform over the tile: it reaches past the first row's diagonal, or starts before the last row's window and is not wholly kept
      if ((col0 + kBKV - 1) > tpos0 || (p.window > 0 && col0 < tpos0 + kBQ - p.window && col0 + kBKV > p.keep)) {
        const int col_limit = rowpos - col0;                               // columns <= col_limit are visible
        const int col_lo = p.window > 0 ? col_limit - p.window + 1 : -(1 << 30);   // and columns >= col_lo
        const int col_keep = p.keep - col0;                                // or < col_keep
#pragma unroll
        for (int c = 0; c < 128; ++c)
          if (c > col_limit || (c < col_lo && c >= col_keep)) r[c] = 0xff800000u;    // -inf
      }
      float mx4[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
#pragma unroll
      for (int c = 0; c < 128; c += 4) {
#pragma unroll
        for (int k = 0; k < 4; ++k) mx4[k] = fmaxf(mx4[k], __uint_as_float(r[c + k]));
      }
      // (rounded up to bf16, the one-tile kernel's reference: the same bits)
      const float mx = __bfloat162float(__float2bfloat16_ru(fmaxf(fmaxf(mx4[0], mx4[1]), fmaxf(mx4[2], mx4[3])))) * p.scale_log2;       // scale > 0
      // the reference maximum only moves by more than 8 (factor 256): P stays within the range of bf16 and fp32 and O is rescaled rarely;
      // O and the running sum share the reference, so the quotient is exact all the same
      const float m_new = (mx > m_run + 8.0f) ? mx : m_run;
      const float base = (m_new == -INFINITY) ? 0.f : m_new;
      const float corr = (m_run == -INFINITY) ? 0.f : fast_exp2(m_run - base);
      if (j > 0 && __any_sync(0xffffffffu, corr != 1.0f)) {
#pragma unroll 1
        for (int c = 0; c < 128; c += 16) {
          uint32_t o[16];
          tmem_ld_32x16(tO + c, o);
          tmem_ld_wait();
#pragma unroll
          for (int k = 0; k < 16; ++k) o[k] = __float_as_uint(__uint_as_float(o[k]) * corr);
          tmem_st_32x16(tO + c, o);
        }
      }
      const uint64_t nbase2 = pair_f32x2(-base, -base);
      uint64_t sum[2] = {0, 0};
#pragma unroll
      for (int c = 0; c < 128; c += 32) {
        uint32_t pk[16];
#pragma unroll
        for (int k = 0; k < 32; k += 2) {
          float e0, e1;
          asm("{\n.reg .b64 x;\nmov.b64 x, {%2, %3};\nfma.rn.f32x2 x, x, %4, %5;\nmov.b64 {%0, %1}, x;\n}"
              : "=f"(e0), "=f"(e1) : "r"(r[c + k]), "r"(r[c + k + 1]), "l"(scale2), "l"(nbase2));
          e0 = fast_exp2(e0);
          e1 = fast_exp2(e1);
          asm("add.rn.f32x2 %0, %0, %1;" : "+l"(sum[c >> 6]) : "l"(pair_f32x2(e0, e1)));
          pk[k >> 1] = pack_bf16(e0, e1);
        }
        tmem_st_32x16(tS + (c >> 1), pk);
      }
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        float s0, s1;
        asm("mov.b64 {%0, %1}, %2;" : "=f"(s0), "=f"(s1) : "l"(sum[h]));
        l_half[h] = l_half[h] * corr + (s0 + s1);
      }
      m_run = m_new;
      tmem_st_wait();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&p_ready[i]);
    }
    // ---- epilogue: O / l, or this share's O, maximum and sum ------------------------------------------
    float l_run = l_half[0] + l_half[1];
    if (ni > 0) ok = ok && mbar_wait_warp(&o_full[i], 0, p.status, kTimeoutTmemFull);
    tc_fence_after();
    const bool row_ok = rows0 + row < q_len;
    const int out_row = q0 + rows0 + row;
    if (ok && splits > 1) {
      float* dst = partial + ((static_cast<size_t>(split) * p.total_q + (row_ok ? out_row : 0)) * p.Hq + head) * (kHD + kPairStat);
#pragma unroll 1
      for (int c = 0; ni > 0 && c < kHD; c += 32) {
        uint32_t o[32];
        tmem_ld_32x32(tO + c, o);
        tmem_ld_wait();
        if (row_ok) {
#pragma unroll
          for (int k = 0; k < 32; k += 2) *reinterpret_cast<float2*>(dst + c + k) = make_float2(__uint_as_float(o[k]), __uint_as_float(o[k + 1]));
        }
      }
      if (row_ok) *reinterpret_cast<float2*>(dst + kHD) = make_float2(m_run, l_run);      // an empty share: -inf, and no O
    } else if (ok && ni > 0) {
      if (p.sink) l_run += exp2f(p.sink[head] * 1.4426950408889634f - (m_run == -INFINITY ? 0.f : m_run));
      float inv = l_run > 0.f ? 1.0f / l_run : 0.f;
      if (p.gate && row_ok) inv /= 1.0f + expf(-__bfloat162float(p.gate[static_cast<size_t>(out_row) * p.gate_ld + head]));
      __nv_bfloat16* orow = p.out + static_cast<size_t>(out_row) * p.ldo + head * kHD;
#pragma unroll 1
      for (int c = 0; c < kHD; c += 32) {
        uint32_t o[32];
        tmem_ld_32x32(tO + c, o);
        tmem_ld_wait();
        if (row_ok) {
#pragma unroll
          for (int k = 0; k < 32; k += 8) {
            uint4 v;
            v.x = pack_bf16(__uint_as_float(o[k]) * inv, __uint_as_float(o[k + 1]) * inv);
            v.y = pack_bf16(__uint_as_float(o[k + 2]) * inv, __uint_as_float(o[k + 3]) * inv);
            v.z = pack_bf16(__uint_as_float(o[k + 4]) * inv, __uint_as_float(o[k + 5]) * inv);
            v.w = pack_bf16(__uint_as_float(o[k + 6]) * inv, __uint_as_float(o[k + 7]) * inv);
            *reinterpret_cast<uint4*>(orow + c + k) = v;
          }
        }
      }
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem, 512);
  }
}

// A warp per (row, head): lane holds four of the 128 values; shares are added in order.
__global__ void __launch_bounds__(256) attn_pair_merge_kernel(const float* __restrict__ partial, const PrefillDev p, int splits) {
  pdl_wait();
  pdl_trigger();
  const long long w = static_cast<long long>(blockIdx.x) * 8 + (threadIdx.x >> 5);
  if (w >= static_cast<long long>(p.total_q) * p.Hq) return;
  const int lane = threadIdx.x & 31, head = static_cast<int>(w % p.Hq);
  const long long t = w / p.Hq;
  const size_t pitch = static_cast<size_t>(p.total_q) * p.Hq * (kHD + kPairStat);
  const float* src = partial + static_cast<size_t>(w) * (kHD + kPairStat);
  float m[kPairSplits], l[kPairSplits], M = -INFINITY;
#pragma unroll
  for (int s = 0; s < kPairSplits; ++s) {
    const float2 st = s < splits ? *reinterpret_cast<const float2*>(src + s * pitch + kHD) : make_float2(-INFINITY, 0.f);
    m[s] = st.x; l[s] = st.y;
    M = fmaxf(M, m[s]);
  }
  float2 a[kPairSplits], b[kPairSplits];
#pragma unroll
  for (int s = 0; s < kPairSplits; ++s) {
    a[s] = b[s] = make_float2(0.f, 0.f);
    if (m[s] != -INFINITY) {                       // a share without a visible key has no O
      a[s] = *reinterpret_cast<const float2*>(src + s * pitch + lane * 4);
      b[s] = *reinterpret_cast<const float2*>(src + s * pitch + lane * 4 + 2);
    }
  }
  float L = 0.f, o[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
  for (int s = 0; s < kPairSplits; ++s) {
    const float f = m[s] == -INFINITY ? 0.f : exp2f(m[s] - M);
    L += l[s] * f;
    o[0] += a[s].x * f; o[1] += a[s].y * f; o[2] += b[s].x * f; o[3] += b[s].y * f;
  }
  if (p.sink) L += exp2f(p.sink[head] * 1.4426950408889634f - (M == -INFINITY ? 0.f : M));
  float inv = L > 0.f ? 1.0f / L : 0.f;
  if (p.gate) inv /= 1.0f + expf(-__bfloat162float(p.gate[t * p.gate_ld + head]));
  *reinterpret_cast<uint2*>(p.out + t * p.ldo + head * kHD + lane * 4) = make_uint2(pack_bf16(o[0] * inv, o[1] * inv), pack_bf16(o[2] * inv, o[3] * inv));
}

template <bool kRope>
static int launch_pair(const CUtensorMap* m, const PrefillDev& p, int num_seqs, int max_q_len, float* partial, int splits, cudaStream_t st) {
  using Cfg = PairCfg<kRope>;
  static std::atomic<unsigned long long> set{0};               // the attribute is the device's
  int dev = 0;
  CAFD_CHECK_CUDA(cudaGetDevice(&dev));
  const unsigned long long bit = 1ull << (dev & 63);
  if (dev > 63 || !(set.load(std::memory_order_relaxed) & bit)) {
    CAFD_CHECK_CUDA(cudaFuncSetAttribute(attn_pair_kernel<kRope>, cudaFuncAttributeMaxDynamicSharedMemorySize, Cfg::kSmem));
    set.fetch_or(bit, std::memory_order_relaxed);
  }
  constexpr int kRows = kRope ? 2 * kBQ : kBQ;
  const dim3 grid(kRope ? p.Hq : p.Hq / 2, (max_q_len + kRows - 1) / kRows, num_seqs * splits);
  launch_pdl(attn_pair_kernel<kRope>, grid, dim3(kPairThreads), Cfg::kSmem, st, m[0], m[1], m[2], m[3], m[4], p, partial, splits);
  if (splits > 1)
    launch_pdl(attn_pair_merge_kernel, dim3(static_cast<unsigned>((static_cast<long long>(p.total_q) * p.Hq + 7) / 8)), dim3(256), 0, st, partial, p,
               splits);
  return static_cast<int>(cudaGetLastError());
}

int attn_pair(const CUtensorMap* maps, const PrefillDev& p, bool rope, int num_seqs, int max_q_len, float* partial, int splits, cudaStream_t st) {
  return rope ? launch_pair<true>(maps, p, num_seqs, max_q_len, partial, splits, st) : launch_pair<false>(maps, p, num_seqs, max_q_len, partial, splits, st);
}

}  // namespace cafd

CAFD_WAIT_LIMIT_SETTER(cafd_attn_pair_set_wait_limit_ns)
