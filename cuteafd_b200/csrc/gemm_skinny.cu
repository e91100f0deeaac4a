// Few rows x large weight: dense projections of at most 32 rows and the routed experts of a decode step, on mma.sync.
//
// Such a product is bound by the bytes of its weights and, at one layer's sizes (17 - 75 MB, 3 - 12 us of HBM), by everything that
// is not streaming them.  The tcgen05 kernel (gemm_tcgen05.cu) pays about 8 us on top: barrier and TMEM set-up, a fill of its ring
// after the previous kernel's end, a 128-row tile whose K range is split over blocks that then meet through scratch, and for the
// experts a plan and a copy of every row into its slab in front of it.  Here
//   * a block of eight warps owns 16 (or 32) weight rows over the whole of K, so nothing is split over blocks; warps split K and meet in
//     shared memory once per tile;
//   * weights go from global memory straight into MMA fragments (a lane's 16 bytes are the A fragments of two m16n8k16 products: both
//     operands use the same permutation of K), 32 KB in flight per block and four blocks per SM at up to eight rows, and the registers of
//     a K group are refilled for the next group, or the next tile, as soon as they are consumed: the stream doesn't stop at tile ends;
//   * weights that no kernel in flight writes are asked for before the programmatic-dependency wait, so that the stream starts under
//     the predecessor (attention, norm, combine) and only the activations are waited for;
//   * the experts read the tokens' rows where they are and write (token, slot) rows: every block sorts the step's routes (at most 256)
//     by expert for itself, which takes the plan and dispatch launches out of a decode step.
// Measured (in a chain with an RMSNorm, graph): 5120 x 2048 at 1 / 8 / 16 rows 5.9 / 6.4 / 8.0 us (tcgen05: 11.2 / 11.5 / 11.9), 2048 x 4096
// 6.8 / 7.2 / 11.4 us (11.0 / 11.5 / 11.9); experts of 128 x (768, 2048), top-8 over random routes, with combine, at 1 / 4 / 8 / 12 rows 28 / 58 / 90 /
// 131 us (with plan and dispatch on tcgen05: 48 / 96 / 136 / 155).  Beyond that the activations' fragments, read once per 16 weight rows,
// fill the L1 pipe and the tcgen05 kernel is the faster one.
// E4M3 weights (128 x 128 block scales) are expanded to f16 in registers and meet the bf16 rows as f16, exactly over the range that matters
// (sk_rows_f16): nothing is quantised, the error of the rows' E4M3 form is gone (logits of the DeepSeek-V3 geometry 1.2e-2 -> 8.7e-3 off
// fp64), and with it two launches per product; a NaN code makes its feature NaN, as it does in the products of larger steps.  Against the
// quantise + tcgen05 E4M3 pair: 24576 x 1536 at 1 / 8 rows behind a norm 12.5 / 13.3 us (19.2 / 19.7), 7168 x 16384 37.7 / 43.4
// (39.8 / 40.5, with the rows' quantisation error); experts of 256 x (2048, 7168), top-8, with combine, at 1 / 4 / 8 rows 91 / 280 / 538 us
// (133 / 337 / 564), 4.2 TB/s where the instructions of the two conversions bound it.
// Sums run in fp32 in a fixed order (K groups of a warp, then warps), so results do not depend on scheduling; they do depend on the
// kernel, so the batch-invariant mode, which promises the same bits at any row count, stays on the tcgen05 kernel.
#include "cafd_api.h"
#include "common.cuh"
#include <atomic>

namespace cafd {

constexpr int kSkThreads = 256;
constexpr int kSkWarps = 8;
constexpr int kSkGroup = 128;              // bytes of a weight row in a K group: one line
constexpr int sk_elems(bool f8) { return f8 ? 128 : 64; }      // K elements of a group (E4M3: one scale block)
constexpr int kSkMaxRows = 32;
constexpr int kSkMaxEntries = 256;         // routes of a step (a thread each)
constexpr int kSkMaxExperts = 512;

bool skinny_takes(const cafd_gemm_args* a);
int skinny_dense(const cafd_gemm_args* a, cudaStream_t st);
int gemm_split_parts(const cafd_gemm_args* a);                    // gemm_split.cu

struct SkinnyDev {
  const uint8_t* w0;             // bf16 or E4M3 rows
  const uint8_t* w1;             // up rows (dual)
  const float* s0;               // E4M3: scale of every 128 x 128 block, [rows / 128, K / 128]
  const float* s1;
  const __nv_bfloat16* x;        // [rows, K]
  void* out;
  const __nv_bfloat16* residual;
  const int* idx;                // grouped: expert of every entry
  int* expert_count;             // grouped: optional, the step's entries per expert are added to it, as the plan of larger steps does
  int K, N, T, ldo, out_f32;
  int n_entries, row_div, E;     // grouped: entry e reads row e / row_div of x and writes row e of out
  int early;                     // the weights (and idx) are not written by the previous kernel of the stream
};

__device__ __forceinline__ uint4 sk_ldw(const uint8_t* p) {      // weights: read once, no L1 allocation
  uint4 v;
  asm volatile("ld.global.nc.L1::no_allocate.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p));
  return v;
}
// Four E4M3 codes -> two f16 pairs, exactly; the NaN codes become NaN.  (bf16 pairs, from shifts and a product with 2^120, cost four
// instructions a pair, as much as this and the rows' conversion together, and turn the NaN codes into +-480; finding the codes beside
// that cost a fifth more.  The experts above took 88 / 265 / 511 us without NaN, 320 / 625 us at 4 / 8 rows with it.)
__device__ __forceinline__ void sk_expand(uint32_t v, uint32_t& lo, uint32_t& hi) {
  asm("{\n.reg .b16 l, h;\nmov.b32 {l, h}, %2;\ncvt.rn.f16x2.e4m3x2 %0, l;\ncvt.rn.f16x2.e4m3x2 %1, h;\n}" : "=r"(lo), "=r"(hi) : "r"(v));
}
// A lane's 32 of the 128 bf16 values of a row that meet an E4M3 block, to f16: times the power of two that brings the largest of the 128
// into [2^14, 2^15), so that everything down to 2^-29 of it keeps all its bits and what is smaller is off by 2^-40 of it at most, less than
// what sums in fp32 lose.  Infinities and NaN stay.  Returns the inverse power.  Lanes 4 g ... 4 g + 3 hold the row.
__device__ __forceinline__ float sk_rows_f16(uint32_t (&x)[16]) {
  uint32_t m[8];
#pragma unroll
  for (int i = 0; i < 8; ++i) asm("max.xorsign.abs.bf16x2 %0, %1, %2;" : "=r"(m[i]) : "r"(x[i]), "r"(x[i + 8]));
#pragma unroll
  for (int d = 4; d; d >>= 1)
#pragma unroll
    for (int i = 0; i < d; ++i) asm("max.xorsign.abs.bf16x2 %0, %0, %1;" : "+r"(m[i]) : "r"(m[i + d]));
  uint32_t top = max((m[0] >> 16) & 0x7fffu, m[0] & 0x7fffu);
  top = max(top, __shfl_xor_sync(0xffffffffu, top, 1));
  top = max(top, __shfl_xor_sync(0xffffffffu, top, 2));
  const uint32_t e = max(top >> 7, 15u);                       // its exponent field
  const uint32_t s = (268u - e) << 7, s2 = s | s << 16;
#pragma unroll
  for (int i = 0; i < 16; ++i) {
    uint32_t t;
    asm("mul.rn.bf16x2 %0, %1, %2;" : "=r"(t) : "r"(x[i]), "r"(s2));
    asm("cvt.rn.f16x2.f32 %0, %1, %2;" : "=r"(x[i]) : "f"(__uint_as_float(t & 0xffff0000u)), "f"(__uint_as_float(t << 16)));
  }
  return __uint_as_float((e - 14u) << 23);
}
__device__ __forceinline__ uint4 sk_ldx(const __nv_bfloat16* p) {      // activations: shared by the SM's blocks through L1
  uint4 v;
  asm volatile("ld.global.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ void sk_mma(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
  asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
               : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
               : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

__device__ __forceinline__ void sk_mma_f16(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
  asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
               : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
               : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

// Kept small: blocks share an SM with the previous kernel's, and what shared memory they need beside it comes off the L1 that serves the
// activations.
struct SkinnyPlan {
  uint16_t act[kSkMaxEntries];       // active experts, ascending, once for every column tile of their entries
  uint16_t off[kSkMaxEntries + 1];   // first place of each one's entries
  uint8_t ent[kSkMaxEntries];        // entries by expert
  int n_act;
};

// Sort the step's routes by expert.  An expert with more entries than `cap` columns is listed again for the rest (a token's routes
// differ, so that takes a row of scores without a number in it, whose slots all name expert 0); which entries a listing holds has to be
// the same in every block, so an expert's entries keep their order.  `tmp`: 2 x kSkMaxExperts ints.
__device__ __forceinline__ void sk_plan(const SkinnyDev& p, SkinnyPlan& s, int* tmp, int cap) {
  int *cnt = tmp, *off = tmp + kSkMaxExperts;
  const int tid = threadIdx.x;
  for (int e = tid; e < p.E; e += kSkThreads) cnt[e] = 0;
  const int mine = tid < p.n_entries ? __ldcg(p.idx + tid) : -1;
  const bool live = mine >= 0 && mine < p.E;       // ids past the stored experts take no row
  __syncthreads();
  int place = 0;
  for (int w = 0; w * 32 < p.n_entries; ++w) {     // 32 entries after 32 entries, so that the order is theirs in every block
    if ((tid >> 5) == w) {
      const unsigned same = __match_any_sync(0xffffffffu, live ? mine : -1);
      const int base = live ? cnt[mine] : 0, before = __popc(same & ((1u << (tid & 31)) - 1u));
      place = base + before;
      __syncwarp();
      if (live && before == 0) cnt[mine] = base + __popc(same);
    }
    __syncthreads();
  }
  if (tid < 32) {
    // lane l: experts [l * per, (l + 1) * per)
    const int per = (p.E + 31) / 32, lo = min(p.E, tid * per), hi = min(p.E, lo + per);
    int n = 0, a = 0;
    for (int e = lo; e < hi; ++e) { n += cnt[e]; a += (cnt[e] + cap - 1) / cap; }
    int in = n, ia = a;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int vn = __shfl_up_sync(0xffffffffu, in, o), va = __shfl_up_sync(0xffffffffu, ia, o);
      if (tid >= o) { in += vn; ia += va; }
    }
    int on = in - n, oa = ia - a;
    for (int e = lo; e < hi; ++e) {
      const int c = cnt[e];
      off[e] = on;
      for (int k = 0; k < c; k += cap) {
        s.act[oa] = static_cast<uint16_t>(e);
        s.off[oa++] = static_cast<uint16_t>(on + k);
      }
      on += c;
    }
    if (tid == 31) { s.n_act = ia; s.off[ia] = static_cast<uint16_t>(in); }
  }
  if (p.expert_count && blockIdx.x == 0)
    for (int e = tid; e < p.E; e += kSkThreads) p.expert_count[e] += cnt[e];
  __syncthreads();
  if (live) s.ent[off[mine] + place] = static_cast<uint8_t>(tid);
  __syncthreads();
}

// kNT: column tiles of 8 rows.  kWK: warps that split K; the other factor of the eight owns row tiles of its own.  kDual: a tile's
// rows 0-7 are gate rows and 8-15 the up rows of the same features.
// kGB: K groups in flight per warp; four where there is at most one tile for each of two blocks per SM.
constexpr int skinny_per_sm(int nt, int gb, bool f8) { return gb > 2 || nt > 2 ? 2 : nt == 1 && !f8 ? 4 : 3; }

template <int kNT, int kWK, int kGB, bool kDual, bool kGrouped, bool kF8>
__global__ void __launch_bounds__(kSkThreads, skinny_per_sm(kNT, kGB, kF8)) skinny_kernel(const SkinnyDev p) {
  constexpr int kWR = kSkWarps / kWK;
  constexpr int kRows = kWR * (kDual ? 8 : 16);    // features of a block's tile
  constexpr int kRS = kNT * 8 + 1;
  constexpr int kElems = sk_elems(kF8);
  // The tensor cores' fp32 sums lose a little with every product they take in: where registers are left, a batch's products are summed
  // apart (2048 x 4096 at eight rows: 4.8e-7 -> 2.4e-7 off fp64, the split sums of the tcgen05 kernel 4.2e-7, at the same time; with more
  // column tiles the sums' registers cost a tenth).  E4M3 blocks are summed apart anyway.
  constexpr bool kApart = !kF8 && kGB > 2 && kNT == 1;
  __shared__ float red[2][kSkWarps * 16 * kRS];
  static_assert(sizeof(red) >= 2 * kSkMaxExperts * sizeof(int), "the sort of the routes works in the reduction buffer");
  __shared__ SkinnyPlan plan;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, q = lane & 3;
  const int wk = warp % kWK, wr = warp / kWK;
  const int K = p.K, groups = K / kElems;
  const size_t pitch = static_cast<size_t>(K) * (kF8 ? 1 : 2);
  const int nb = (groups + kWK * kGB - 1) / (kWK * kGB);       // batches of a tile
  const int per_expert = (p.N + kRows - 1) / kRows;

  if (!p.early) { pdl_wait(); pdl_trigger(); }
  int n_tiles = per_expert;
  if (kGrouped) {
    sk_plan(p, plan, reinterpret_cast<int*>(red[0]), kNT * 8);
    n_tiles = plan.n_act * per_expert;
  }
  const float *sc0 = nullptr, *sc1 = nullptr;                  // E4M3: scales of the next tile's rows
  auto rows_of = [&](int tile, const uint8_t*& r0, const uint8_t*& r1) {
    size_t base = 0;
    int f = tile;
    if (kGrouped) {
      const int a = tile / per_expert;
      f = tile - a * per_expert;
      base = static_cast<size_t>(plan.act[a]) * p.N;
    }
    const int row = f * kRows + wr * (kDual ? 8 : 16) + g;     // rows past the end repeat the last one and are never stored
    const size_t n0 = base + min(row, p.N - 1);
    r0 = p.w0 + n0 * pitch + q * 16;
    r1 = kDual ? p.w1 + n0 * pitch + q * 16 : p.w0 + (base + min(row + 8, p.N - 1)) * pitch + q * 16;
    if (kF8) {                                                 // N is a multiple of 128: a tile lies within one row of blocks
      sc0 = p.s0 + n0 / 128 * groups;
      sc1 = kDual ? p.s1 + n0 / 128 * groups : sc0;
    }
  };
  uint4 a[kGB][2][2];                                          // [group][row half][64-byte half of the group]
  float sc[kGB][2];
  auto fetch = [&](int i, int b, const uint8_t* r0, const uint8_t* r1) {
    const int grp = (b * kGB + i) * kWK + wk;
    if (grp < groups) {
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        a[i][0][h] = sk_ldw(r0 + grp * kSkGroup + h * 64);
        a[i][1][h] = sk_ldw(r1 + grp * kSkGroup + h * 64);
      }
      if (kF8) {
        sc[i][0] = __ldg(sc0 + grp);
        sc[i][1] = kDual ? __ldg(sc1 + grp) : sc[i][0];
      }
    }
  };
  int tile = blockIdx.x;
  const uint8_t *r0 = p.w0, *r1 = p.w0;
  if (tile < n_tiles) {
    rows_of(tile, r0, r1);
#pragma unroll
    for (int i = 0; i < kGB; ++i) fetch(i, 0, r0, r1);
  }
  if (p.early) { pdl_wait(); pdl_trigger(); }

  for (int turn = 0; tile < n_tiles; tile += gridDim.x, ++turn) {
    int f = tile, cols = p.T, first = 0;
    if (kGrouped) {
      const int ord = tile / per_expert;
      f = tile - ord * per_expert;
      first = plan.off[ord];
      cols = plan.off[ord + 1] - first;
    }
    const __nv_bfloat16* xr[kNT];
#pragma unroll
    for (int nt = 0; nt < kNT; ++nt) {
      const int c = min(nt * 8 + g, cols - 1);                 // columns past the end repeat the last one
      const int row = kGrouped ? plan.ent[first + c] / p.row_div : c;
      xr[nt] = p.x + static_cast<size_t>(row) * K + q * (kF8 ? 16 : 8);
    }
    float acc[kNT][4];
#pragma unroll
    for (int nt = 0; nt < kNT; ++nt) acc[nt][0] = acc[nt][1] = acc[nt][2] = acc[nt][3] = 0.f;
    float sum[4] = {0.f, 0.f, 0.f, 0.f};
    const int next = tile + gridDim.x;
    for (int b = 0; b < nb; ++b) {
      const bool last = b + 1 == nb;
      if (last && next < n_tiles) rows_of(next, r0, r1);
#pragma unroll
      for (int i = 0; i < kGB; ++i) {
        const int grp = (b * kGB + i) * kWK + wk;
        if (grp < groups) {
#pragma unroll
          for (int nt = 0; nt < kNT; ++nt) {
            if (nt * 8 < cols) {
              const __nv_bfloat16* xg = xr[nt] + grp * kElems;
              if constexpr (kF8) {
                // a block's products are summed apart and scaled once
                uint32_t xb[16];
#pragma unroll
                for (int h = 0; h < 4; ++h) {
                  const uint4 v = sk_ldx(xg + (h >> 1) * 64 + (h & 1) * 8);
                  xb[4 * h] = v.x; xb[4 * h + 1] = v.y; xb[4 * h + 2] = v.z; xb[4 * h + 3] = v.w;
                }
                const float inv = sk_rows_f16(xb);
                const float i0 = __shfl_sync(0xffffffffu, inv, 8 * q), i1 = __shfl_sync(0xffffffffu, inv, 8 * q + 4);     // rows 2 q, 2 q + 1
                float raw[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                  const uint32_t w0[4] = {a[i][0][h].x, a[i][0][h].y, a[i][0][h].z, a[i][0][h].w};
                  const uint32_t w1[4] = {a[i][1][h].x, a[i][1][h].y, a[i][1][h].z, a[i][1][h].w};
#pragma unroll
                  for (int e = 0; e < 4; ++e) {
                    uint32_t a0, a1, a2, a3;
                    sk_expand(w0[e], a0, a2);
                    sk_expand(w1[e], a1, a3);
                    sk_mma_f16(raw, a0, a1, a2, a3, xb[8 * h + 2 * e], xb[8 * h + 2 * e + 1]);
                  }
                }
                acc[nt][0] += raw[0] * i0 * sc[i][0];
                acc[nt][1] += raw[1] * i1 * sc[i][0];
                acc[nt][2] += raw[2] * i0 * sc[i][1];
                acc[nt][3] += raw[3] * i1 * sc[i][1];
              } else {
                const uint4 b0 = sk_ldx(xg), b1 = sk_ldx(xg + 32);
                sk_mma(acc[nt], a[i][0][0].x, a[i][1][0].x, a[i][0][0].y, a[i][1][0].y, b0.x, b0.y);
                sk_mma(acc[nt], a[i][0][0].z, a[i][1][0].z, a[i][0][0].w, a[i][1][0].w, b0.z, b0.w);
                sk_mma(acc[nt], a[i][0][1].x, a[i][1][1].x, a[i][0][1].y, a[i][1][1].y, b1.x, b1.y);
                sk_mma(acc[nt], a[i][0][1].z, a[i][1][1].z, a[i][0][1].w, a[i][1][1].w, b1.z, b1.w);
              }
            }
          }
        }
        if (!last) fetch(i, b + 1, r0, r1);
        else if (next < n_tiles) fetch(i, 0, r0, r1);
      }
      if constexpr (kApart) {
#pragma unroll
        for (int e = 0; e < 4; ++e) { sum[e] += acc[0][e]; acc[0][e] = 0.f; }
      }
    }
    // warps meet: buffer turn & 1 was last read two tiles ago, before the barrier of the tile between
    float* rb = red[turn & 1];
    float* mine = rb + warp * 16 * kRS + 2 * q;
#pragma unroll
    for (int nt = 0; nt < kNT; ++nt) {
      if (nt * 8 < cols) {
        const float(&v)[4] = kApart ? sum : acc[nt];
        mine[g * kRS + nt * 8] = v[0];
        mine[g * kRS + nt * 8 + 1] = v[1];
        mine[(g + 8) * kRS + nt * 8] = v[2];
        mine[(g + 8) * kRS + nt * 8 + 1] = v[3];
      }
    }
    __syncthreads();
    for (int o = tid; o < kRows * cols; o += kSkThreads) {
      const int col = o / kRows, r = o % kRows, feat = f * kRows + r;
      if (feat >= p.N) continue;
      const int tr = kDual ? r & 7 : r & 15, own = (kDual ? r >> 3 : r >> 4) * kWK;
      float v = 0.f, u = 0.f;
#pragma unroll
      for (int w = 0; w < kWK; ++w) {
        v += rb[((own + w) * 16 + tr) * kRS + col];
        if (kDual) u += rb[((own + w) * 16 + tr + 8) * kRS + col];
      }
      if (kDual) v = silu(v) * u;
      const size_t at = static_cast<size_t>(kGrouped ? plan.ent[first + col] : col) * p.ldo + feat;
      if (p.out_f32) {
        reinterpret_cast<float*>(p.out)[at] = v;
      } else {
        if (p.residual) v += __bfloat162float(p.residual[at]);
        reinterpret_cast<__nv_bfloat16*>(p.out)[at] = __float2bfloat16(v);
      }
    }
  }
}

template <int kNT, int kWK, int kGB, bool kDual, bool kGrouped, bool kF8>
static int launch_skinny(const SkinnyDev& p, long long tiles, int sms, cudaStream_t st) {
  // Left to itself the driver sizes shared memory for this kernel alone.  The first blocks then start on SMs that the previous
  // kernel still holds at another split, a fourth block finds no room until an SM is drained, and its share of the tiles runs after
  // everybody else's (fc1 of eight rows: 83 us in the chain, 55 us alone).  64 KB hold four blocks of one column
  // tile, three of two and one of four (whose products have at most one tile per SM) and leave the rest to L1.  The attribute is the
  // device's: it is set once on each.
  static std::atomic<unsigned long long> set{0};
  int dev = 0;
  CAFD_CHECK_CUDA(cudaGetDevice(&dev));
  const unsigned long long bit = 1ull << (dev & 63);
  if (dev > 63 || !(set.load(std::memory_order_relaxed) & bit)) {
    CAFD_CHECK_CUDA(cudaFuncSetAttribute(skinny_kernel<kNT, kWK, kGB, kDual, kGrouped, kF8>, cudaFuncAttributePreferredSharedMemoryCarveout, 28));
    set.fetch_or(bit, std::memory_order_relaxed);
  }
  const long long most = static_cast<long long>(skinny_per_sm(kNT, kGB, kF8)) * sms;
  launch_pdl(skinny_kernel<kNT, kWK, kGB, kDual, kGrouped, kF8>, dim3(static_cast<unsigned>(tiles < most ? tiles : most)), dim3(kSkThreads), 0, st, p);
  return static_cast<int>(cudaGetLastError());
}

// At most 16 groups (K 1024, E4M3 2048) keep eight K-splitting warps half idle: four of them then, and two row tiles per block.
template <int kNT, bool kDual, bool kGrouped, bool kF8 = false>
static int pick_skinny(const SkinnyDev& p, long long max_experts, int sms, cudaStream_t st) {
  const bool wide = p.K > 16 * sk_elems(kF8);
  const int feats = (wide ? 1 : 2) * (kDual ? 8 : 16);
  const long long tiles = max_experts * ((p.N + feats - 1) / feats);
  if (!wide) return launch_skinny<kNT, 4, 2, kDual, kGrouped, kF8>(p, tiles, sms, st);
  if constexpr (!kGrouped && kNT <= 2)
    if (tiles <= 2 * sms) return launch_skinny<kNT, 8, 4, kDual, kGrouped, kF8>(p, tiles, sms, st);
  return launch_skinny<kNT, 8, 2, kDual, kGrouped, kF8>(p, tiles, sms, st);
}

static int sm_count() {
  int dev = 0, sms = 148;
  if (cudaGetDevice(&dev) == cudaSuccess) cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  return sms;
}
static bool aligned16(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15u) == 0; }

}  // namespace cafd

using namespace cafd;

// Whether cafd_gemm hands a dense product to this kernel.  Up to eight rows and K 4096 it is the faster one at every size measured up to some
// 200 M weights (100 M of a gate and up pair): 2048 x 4096 to 65536 x 1024, 32000 x 4096 52 - 55 against 55 us, 10944 x 4096 pairs 40 - 43
// against 42 us; beyond, the other kernel's copies keep more bytes in flight and its fill is not seen: 151936 x 2048 109 against 105 us,
// 14336 x 4096 pairs 52 - 57 against 49 us.  Longer K: one wave of tiles with four groups in flight (2176 x 7168: 11.8 against 13.3 us);
// beyond it the rows of x don't stay in L1 (18432 x 7168 gate and up: 106 against 91 us).  Nine to sixteen rows: up to K 4096 and one wave of
// tiles (5120 x 2048: 8.0 against 11.9 us; but 37984 x 2048: 42 against 38 us, 2176 x 7168: 19 against 14 us).  Up to 32 rows: a tile per
// SM at most, where the other kernel cuts K nine ways and one block adds the parts (2048 x 4096: 13 against 31 us behind decode attention;
// behind a norm 15 against 17 us at 17 rows, 19 against 18 at 32; 5120 x 2048: 15.6 against 15.1 us).
bool cafd::skinny_takes(const cafd_gemm_args* a) {
  const int sms = a->num_sms > 0 ? a->num_sms : sm_count();
  const int tiles = (a->n_features + (a->dual ? 7 : 15)) / (a->dual ? 8 : 16);
  const long long weights = static_cast<long long>(a->n_features) * a->k;        // of one of the two where there is a pair
  const bool rows = a->x_rows <= 8 ? (a->k <= 4096 ? weights <= (a->dual ? 50 : 200) * 1000000ll : tiles <= 2 * sms)
                                   : a->x_rows <= kSkMaxRows && a->k <= 4096 && tiles <= (a->x_rows <= 16 ? 4 : 1) * sms;
  // tiles of 128 features whose K a cluster shares: 2048 x 4096 at 9 / 17 / 32 rows 8.2 / 13.1 / 17.1 us here, 5.7 / 6.7 / 7.6 there, 256 /
  // 1024 x 7168 at 8 rows 10.0 / 10.7 and 4.2 / 5.8 (but 128 x 2048 at 10 rows 3.3 here)
  if ((a->x_rows > 16 || (a->k >= 4096 && tiles <= sms)) && gemm_split_parts(a)) return false;
  return a->swap && !a->fp8 && a->x_rows > 0 && rows && a->k % sk_elems(false) == 0 && !a->tile_expert && !a->row_dst &&
         !a->row_scale && !a->wait_flag && !a->signal_flag && !a->rs_ranks && !a->n_signal_flags && !(a->dual && a->glu) &&
         !(a->dual && (!a->w1 || a->w1_row_offset)) && fixed_kv_split_tokens() == 0 && aligned16(a->w0) && aligned16(a->w1) && aligned16(a->x);
}

extern "C" int cafd_gemm_few_rows(const cafd_gemm_args* a) { return a && skinny_takes(a); }

int cafd::skinny_dense(const cafd_gemm_args* a, cudaStream_t st) {
  SkinnyDev p{};
  p.w0 = static_cast<const uint8_t*>(a->w0);
  p.w1 = static_cast<const uint8_t*>(a->w1);
  p.x = static_cast<const __nv_bfloat16*>(a->x);
  p.out = a->out;
  p.residual = static_cast<const __nv_bfloat16*>(a->residual);
  p.K = a->k; p.N = a->n_features; p.T = a->x_rows; p.ldo = a->ldo; p.out_f32 = a->out_f32;
  p.row_div = 1;
  p.early = a->w_resident;
  const int sms = a->num_sms > 0 ? a->num_sms : sm_count();
  if (p.T <= 8) return a->dual ? pick_skinny<1, true, false>(p, 1, sms, st) : pick_skinny<1, false, false>(p, 1, sms, st);
  if (p.T <= 16) return a->dual ? pick_skinny<2, true, false>(p, 1, sms, st) : pick_skinny<2, false, false>(p, 1, sms, st);
  return a->dual ? pick_skinny<4, true, false>(p, 1, sms, st) : pick_skinny<4, false, false>(p, 1, sms, st);
}

extern "C" int cafd_moe_skinny_max_entries(void) { return kSkMaxEntries; }

// Routed experts of a decode step without plan or slab: entry e = (token, slot) with expert idx[e] reads row e / row_div of x and writes
// row e of out (entries with an id outside [0, E) write nothing).  w [E, N, K]; w_up: silu(x w^T) * (x w_up^T).  s / s_up not null: w and
// w_up are E4M3 with a scale for every 128 x 128 block, [E, N / 128, K / 128], and x stays bf16.  At most cafd_moe_skinny_max_entries()
// entries; an expert with distinct tokens has at most max_per_expert (<= 16; E4M3 <= 8), more of them are done in several goes.  early: idx and the weights are not written by the previous
// kernel in the stream.
extern "C" int cafd_moe_skinny(const void* x, int row_div, const void* w, const void* w_up, const float* s, const float* s_up, const int* idx,
                               int n_entries, int max_per_expert, int E, int K, int N, void* out, int ldo, int* expert_count, int early,
                               int num_sms, cafd_stream_t stream) {
  if (n_entries <= 0) return 0;
  const int unit = sk_elems(s != nullptr);
  if (n_entries > kSkMaxEntries || (early && expert_count) || E < 1 || E > kSkMaxExperts || K < unit || K % unit || N < 1 || row_div < 1 ||
      max_per_expert < 1 || max_per_expert > (s ? 8 : 16) || (s && (N % 128 || (w_up && !s_up))) || !aligned16(x) || !aligned16(w) || !aligned16(w_up))
    return -10;
  SkinnyDev p{};
  p.w0 = static_cast<const uint8_t*>(w);
  p.w1 = static_cast<const uint8_t*>(w_up);
  p.s0 = s; p.s1 = s_up;
  p.x = static_cast<const __nv_bfloat16*>(x);
  p.out = out;
  p.idx = idx;
  p.expert_count = expert_count;
  p.K = K; p.N = N; p.ldo = ldo; p.E = E;
  p.n_entries = n_entries; p.row_div = row_div; p.early = early;
  const int most = n_entries < E ? n_entries : E, sms = num_sms > 0 ? num_sms : sm_count();
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  if (s) return w_up ? pick_skinny<1, true, true, true>(p, most, sms, st) : pick_skinny<1, false, true, true>(p, most, sms, st);
  if (max_per_expert <= 8) return w_up ? pick_skinny<1, true, true>(p, most, sms, st) : pick_skinny<1, false, true>(p, most, sms, st);
  return w_up ? pick_skinny<2, true, true>(p, most, sms, st) : pick_skinny<2, false, true>(p, most, sms, st);
}

// out [T, N] = x [T, K] w^T (+ residual) for at most eight bf16 rows and E4M3 weights with a scale for every 128 x 128 block; w_up: SwiGLU pair.
extern "C" int cafd_linear_w8(const void* x, int T, const void* w, const void* w_up, const float* s, const float* s_up, int K, int N, void* out,
                              int ldo, const void* residual, int early, int num_sms, cafd_stream_t stream) {
  if (T <= 0) return 0;
  if (T > 8 || K < 128 || K % 128 || N < 128 || N % 128 || !s || (w_up && !s_up) || !aligned16(x) || !aligned16(w) || !aligned16(w_up)) return -10;
  SkinnyDev p{};
  p.w0 = static_cast<const uint8_t*>(w);
  p.w1 = static_cast<const uint8_t*>(w_up);
  p.s0 = s; p.s1 = s_up;
  p.x = static_cast<const __nv_bfloat16*>(x);
  p.out = out;
  p.residual = static_cast<const __nv_bfloat16*>(residual);
  p.K = K; p.N = N; p.T = T; p.ldo = ldo; p.row_div = 1; p.early = early;
  const int sms = num_sms > 0 ? num_sms : sm_count();
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  return w_up ? pick_skinny<1, true, false, true>(p, 1, sms, st) : pick_skinny<1, false, false, true>(p, 1, sms, st);
}
