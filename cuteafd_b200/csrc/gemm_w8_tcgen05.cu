// Expert-grouped E4M3 weights (128 x 128 block scales) x bf16 rows on tcgen05, for steps of more rows than the few-row kernel takes.
//
// Bound: the stored bytes of the experts (a prompt touches all of them) and, close behind, the expansion of every code.  The form this
// replaces expanded a layer's experts to bf16 in memory and ran the bf16 kernel over them: five bytes of traffic for every stored byte.
// Here a code leaves memory once and is expanded on its way to the tensor cores, each value float(code) * scale rounded to bf16, the bits
// that cafd_fp8_dequant_block128 writes:
//
//   warp 0       TMA producer of the row tile (rows on the MMA N side, kBX of them, 128 of K per stage)
//   warp 1       MMA issuer
//   warp 2       TMA producer of the stored weights: a ring of raw 128 x 128-byte tiles, so that bytes in flight cover the latency of HBM
//   warp 3       TMEM owner
//   warps 4-7    epilogue: thread = feature, two features of two rows are exchanged between lanes so that a store is four bytes
//   warps 8-23   weight decoders, eight warps per weight tile, thread = half of a weight row: 64 codes from the raw ring to 32 TMEM columns
//
// A unit is two weight tiles of 128 features (gate and up, or two neighbours) x kBX rows.  The expanded weights are the MMA's A operand in
// TMEM, not in shared memory: a K block of 128 x 128 weights meets 128 rows in 512 cycles, of which the tensor core's reads of the rows take
// 256 of shared memory's; written to and read back from shared memory the weights would take 512 more.  TMEM: accumulators in columns 0-255
// (two buffers up to 64 rows, one of 128 rows, which the epilogue empties into registers before it stores anything), two stages of two
// expanded tiles in 256-511.
//
// Reference counterpart: native/shared/include/cuteafd_fp8_moe.h:14-76 (the exported block-scaled expert programs).
#include "cafd_api.h"
#include "common.cuh"
#include "host_tma.h"

#include <atomic>

namespace cafd {

constexpr int kW8BK = 128;                 // K per stage: one scale block, 128 bytes of a weight row
constexpr int kW8Threads = 768;
constexpr int kW8Decoders = 16;            // warps
// Registers per thread: launched with 80 (768 threads: six warpgroups, 480 in all), the epilogue keeps a unit's results in them.
constexpr int kW8RegsControl = 40, kW8RegsEpilogue = 152, kW8RegsDecode = 72;
static_assert(kW8RegsControl + kW8RegsEpilogue + kW8Decoders / 4 * kW8RegsDecode <= 80 * kW8Threads / 128, "the launch's registers");
constexpr int kW8Tile = 128 * kW8BK;       // stored bytes of a weight tile and stage
constexpr int kW8Raw = 4;                  // stages of the raw ring, two tiles each

struct W8Dev {
  const float* s0;             // [experts * N / 128, K / 128]
  const float* s1;
  __nv_bfloat16* out;
  const int* row_dst;
  const int* tile_expert;
  const int* tile_row0;
  const int* num_x_tiles;
  const uint32_t* wait_flag;
  const uint32_t* epoch;
  uint32_t* done_counter;
  uint32_t* signal_flag;
  uint32_t* status;
  int nkb, n_features, ldo, w_rows_per_expert, w_units, max_x_tiles;
};

template <int kBX>
struct W8Cfg {
  static constexpr int kXHalf = kBX * 128;                       // kBX rows x 64 bf16
  static constexpr int kXBytes = 2 * kXHalf;
  static constexpr int kXStages = kBX == 128 ? 3 : kBX == 64 ? 5 : 8;
  static constexpr int kAccBufs = kBX == 128 ? 1 : 2;
  static constexpr int kSmem = kW8Raw * 2 * kW8Tile + kXStages * kXBytes + 1024;
  static_assert(kAccBufs * 2 * kBX <= 256, "accumulators end where the expanded weights begin");
  static_assert(kSmem <= 227 * 1024 - 512, "shared memory");
};

// Four codes -> two bf16 pairs of float(code) * s: the conversion to f16 and on to fp32 is exact, so each value is rounded once.
__device__ __forceinline__ void w8_expand(uint32_t v, uint64_t s2, uint32_t& lo, uint32_t& hi) {
  asm("{\n.reg .b16 p, q, a, b, c, d;\n.reg .b32 x, y;\n.reg .f32 e, f, g, h;\n.reg .b64 m, n;\n"
      "mov.b32 {p, q}, %2;\n"
      "cvt.rn.f16x2.e4m3x2 x, p;\ncvt.rn.f16x2.e4m3x2 y, q;\n"
      "mov.b32 {a, b}, x;\nmov.b32 {c, d}, y;\n"
      "cvt.f32.f16 e, a;\ncvt.f32.f16 f, b;\ncvt.f32.f16 g, c;\ncvt.f32.f16 h, d;\n"
      "mov.b64 m, {e, f};\nmov.b64 n, {g, h};\n"
      "mul.rn.f32x2 m, m, %3;\nmul.rn.f32x2 n, n, %3;\n"
      "mov.b64 {e, f}, m;\nmov.b64 {g, h}, n;\n"
      "cvt.rn.bf16x2.f32 %0, f, e;\ncvt.rn.bf16x2.f32 %1, h, g;\n}"
      : "=r"(lo), "=r"(hi) : "r"(v), "l"(s2));
}

template <bool kDual, int kBX>
__global__ void __launch_bounds__(kW8Threads, 1)
gemm_w8_kernel(const __grid_constant__ CUtensorMap tm_x, const __grid_constant__ CUtensorMap tm_w0,
               const __grid_constant__ CUtensorMap tm_w1, const W8Dev p) {
  using Cfg = W8Cfg<kBX>;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* raw = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t* sx = raw + kW8Raw * 2 * kW8Tile;
  __shared__ uint64_t raw_full[kW8Raw], raw_empty[kW8Raw], x_full[Cfg::kXStages], x_empty[Cfg::kXStages];
  __shared__ uint64_t a_full[2], a_empty[2], acc_full[2], acc_empty[2];
  __shared__ uint32_t tmem_slot;
  __shared__ int s_tiles;
  const int warp = warp_uniform(threadIdx.x >> 5), lane = threadIdx.x & 31;

  if (threadIdx.x == 0) {
    for (int i = 0; i < kW8Raw; ++i) { mbar_init(&raw_full[i], 1); mbar_init(&raw_empty[i], kW8Decoders); }
    for (int i = 0; i < Cfg::kXStages; ++i) { mbar_init(&x_full[i], 1); mbar_init(&x_empty[i], 1); }
    for (int i = 0; i < 2; ++i) {
      mbar_init(&a_full[i], kW8Decoders); mbar_init(&a_empty[i], 1);
      mbar_init(&acc_full[i], 1); mbar_init(&acc_empty[i], 128);
    }
    mbar_fence_init();
    pdl_wait();
    bool ok = true;
    if (p.wait_flag) {
      ok = wait_flag_ge(p.wait_flag, *p.epoch, p.status);
      asm volatile("fence.proxy.async;" ::: "memory");      // a peer's ordinary stores, read by TMA
    }
    s_tiles = ok ? min(*reinterpret_cast<const volatile int*>(p.num_x_tiles), p.max_x_tiles) : 0;
  }
  if (warp == 3) {
    tmem_alloc(&tmem_slot, 512);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  pdl_wait();
  pdl_trigger();
  const uint32_t tmem = tmem_slot;
  const int units = s_tiles * p.w_units, nkb = p.nkb;
  // Neighbouring blocks take the weight tiles of one row tile: its rows come out of L2, its weights are read once.
  auto tile_of = [&](int unit, int t, int expert) {          // first weight row of tile t of the unit (past an odd count: the tile before)
    const int wu = unit % p.w_units;
    int f = kDual ? wu * 128 : wu * 256 + t * 128;
    if (f >= p.n_features) f -= 128;
    return expert * p.w_rows_per_expert + f;
  };

  if (warp < 4) reg_dec<kW8RegsControl>();
  if (warp == 0) {
    if (lane == 0) {
      tma_prefetch_desc(&tm_x);
      int st = 0;
      uint32_t ph = 0;
      bool ok = true;
      for (int u = blockIdx.x; ok && u < units; u += gridDim.x) {
        const int row0 = p.tile_row0[u / p.w_units];
        for (int kb = 0; kb < nkb; ++kb) {
          if (!mbar_wait(&x_empty[st], ph ^ 1, p.status, kTimeoutEmptyBarrier)) { ok = false; break; }
          uint8_t* d = sx + st * Cfg::kXBytes;
          mbar_expect_tx(&x_full[st], Cfg::kXBytes);
          tma_load_2d(d, &tm_x, &x_full[st], kb * kW8BK, row0);
          tma_load_2d(d + Cfg::kXHalf, &tm_x, &x_full[st], kb * kW8BK + 64, row0);
          if (++st == Cfg::kXStages) { st = 0; ph ^= 1; }
        }
      }
    }
  } else if (warp == 1) {
    constexpr uint32_t idesc = make_idesc(128, kBX, 1, 1);
    const uint64_t xdesc = smem_desc_k_sw128(smem_u32(sx));
    int st = 0, n = 0, it = 0;
    uint32_t ph = 0;
    bool ok = true;
    for (int u = blockIdx.x; ok && u < units; u += gridDim.x, ++n) {
      const int buf = n % Cfg::kAccBufs;
      if (!mbar_wait_warp(&acc_empty[buf], ((n / Cfg::kAccBufs) & 1) ^ 1, p.status, kTimeoutTmemEmpty)) { ok = false; break; }
      const uint32_t d0 = tmem + buf * 2 * kBX;
      for (int kb = 0; kb < nkb; ++kb, ++it) {
        const int as = it & 1;
        if (!mbar_wait_warp(&x_full[st], ph, p.status, kTimeoutFullBarrier) ||
            !mbar_wait_warp(&a_full[as], (it >> 1) & 1, p.status, kTimeoutFullBarrier)) { ok = false; break; }
        tc_fence_after();
        if (elect_one()) {
          const uint64_t x0 = xdesc + static_cast<uint64_t>(st * (Cfg::kXBytes >> 4));
          const uint32_t a0 = tmem + 256 + as * 128;
#pragma unroll
          for (int t = 0; t < 2; ++t)
#pragma unroll
            for (int k = 0; k < 8; ++k)
              umma_f16_ts(d0 + t * kBX, a0 + t * 64 + k * 8, x0 + (((k >> 2) * Cfg::kXHalf + (k & 3) * 32) >> 4), idesc, (kb | k) ? 1u : 0u);
          umma_commit(&a_empty[as]);
          umma_commit(&x_empty[st]);
          if (kb == nkb - 1) umma_commit(&acc_full[buf]);
        }
        __syncwarp();
        if (++st == Cfg::kXStages) { st = 0; ph ^= 1; }
      }
    }
  } else if (warp == 2) {
    if (lane == 0) {
      tma_prefetch_desc(&tm_w0);
      if (kDual) tma_prefetch_desc(&tm_w1);
      int st = 0;
      uint32_t ph = 0;
      bool ok = true;
      for (int u = blockIdx.x; ok && u < units; u += gridDim.x) {
        const int expert = p.tile_expert[u / p.w_units], r0 = tile_of(u, 0, expert), r1 = tile_of(u, 1, expert);
        for (int kb = 0; kb < nkb; ++kb) {
          if (!mbar_wait(&raw_empty[st], ph ^ 1, p.status, kTimeoutEmptyBarrier)) { ok = false; break; }
          uint8_t* d = raw + st * 2 * kW8Tile;
          mbar_expect_tx(&raw_full[st], 2 * kW8Tile);
          tma_load_2d(d, &tm_w0, &raw_full[st], kb * kW8BK, r0);
          tma_load_2d(d + kW8Tile, kDual ? &tm_w1 : &tm_w0, &raw_full[st], kb * kW8BK, r1);
          if (++st == kW8Raw) { st = 0; ph ^= 1; }
        }
      }
    }
  } else if (warp >= 8) {
    // ------------------------------------------------------------------ weight decoders
    reg_dec<kW8RegsDecode>();
    const int t = ((warp - 8) >> 2) & 1, h = (warp - 8) >> 3, r = (warp & 3) * 32 + lane;
    const uint32_t lanes = static_cast<uint32_t>((warp & 3) * 32) << 16;
    int st = 0, it = 0;
    uint32_t ph = 0;
    bool ok = true;
    for (int u = blockIdx.x; ok && u < units; u += gridDim.x) {
      const float* sc = (kDual && t ? p.s1 : p.s0) + static_cast<size_t>(tile_of(u, t, p.tile_expert[u / p.w_units]) / 128) * nkb;
      float s = __ldg(sc);
      for (int kb = 0; kb < nkb; ++kb, ++it) {
        const int as = it & 1;
        uint64_t s2;
        asm("mov.b64 %0, {%1, %1};" : "=l"(s2) : "f"(s));
        if (kb + 1 < nkb) s = __ldg(sc + kb + 1);
        if (!mbar_wait_warp(&raw_full[st], ph, p.status, kTimeoutFullBarrier)) { ok = false; break; }
        const uint8_t* row = raw + (st * 2 + t) * kW8Tile + r * 128;
        uint4 v[4];
#pragma unroll
        for (int c = 0; c < 4; ++c) v[c] = *reinterpret_cast<const uint4*>(row + (((h * 4 + c) ^ (r & 7)) << 4));
        uint32_t o[32];
#pragma unroll
        for (int c = 0; c < 4; ++c) {
          w8_expand(v[c].x, s2, o[c * 8 + 0], o[c * 8 + 1]);
          w8_expand(v[c].y, s2, o[c * 8 + 2], o[c * 8 + 3]);
          w8_expand(v[c].z, s2, o[c * 8 + 4], o[c * 8 + 5]);
          w8_expand(v[c].w, s2, o[c * 8 + 6], o[c * 8 + 7]);
        }
        __syncwarp();
        if (lane == 0) mbar_arrive(&raw_empty[st]);
        if (++st == kW8Raw) { st = 0; ph ^= 1; }
        if (!mbar_wait_warp(&a_empty[as], ((it >> 1) & 1) ^ 1, p.status, kTimeoutEmptyBarrier)) { ok = false; break; }
        tc_fence_after();
        tmem_st_32x32(tmem + lanes + 256 + as * 128 + t * 64 + h * 32, o);
        tmem_st_wait();
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(&a_full[as]);
      }
    }
  } else if (warp >= 4) {
    // ------------------------------------------------------------------ epilogue: thread = feature
    reg_inc<kW8RegsEpilogue>();
    const int quad = warp & 3;
    constexpr int kTiles = kDual ? 1 : 2;                    // 128-feature tiles of results
    int n = 0;
    bool ok = true;
    for (int u = blockIdx.x; ok && u < units; u += gridDim.x, ++n) {
      const int xt = u / p.w_units, wu = u % p.w_units, row0 = p.tile_row0[xt];
      int dst[(kBX + 31) / 32];                              // where rows lane, lane + 32, ... go
#pragma unroll
      for (int i = 0; i < (kBX + 31) / 32; ++i) {
        const int row = row0 + i * 32 + lane;
        dst[i] = p.row_dst ? p.row_dst[row] : row;
      }
      const int buf = n % Cfg::kAccBufs;
      if (!mbar_wait_warp(&acc_full[buf], (n / Cfg::kAccBufs) & 1, p.status, kTimeoutTmemFull)) { ok = false; break; }
      tc_fence_after();
      const uint32_t t0 = tmem + (static_cast<uint32_t>(quad * 32) << 16) + buf * 2 * kBX;
      auto store = [&](int f, int j, uint32_t mine) {        // mine: this lane's feature of rows j and j + 1
        const uint32_t other = __shfl_xor_sync(0xffffffffu, mine, 1);
        const uint32_t v = lane & 1 ? __byte_perm(other, mine, 0x7632) : __byte_perm(mine, other, 0x5410);
        const int d0 = __shfl_sync(0xffffffffu, dst[j >> 5], j & 31), d1 = __shfl_sync(0xffffffffu, dst[j >> 5], (j + 1) & 31);
        const int d = lane & 1 ? d1 : d0;
        if (d >= 0) *reinterpret_cast<uint32_t*>(p.out + static_cast<size_t>(d) * p.ldo + (f & ~1)) = v;
      };
      uint32_t v[kTiles][kBX / 2];                           // rows 2 i and 2 i + 1 of this thread's feature
#pragma unroll
      for (int c = 0; c < kBX; c += 16) {
        uint32_t g[16], h[16];
        tmem_ld_32x16(t0 + c, g);
        tmem_ld_32x16(t0 + kBX + c, h);
        tmem_ld_wait();
#pragma unroll
        for (int j = 0; j < 16; j += 2) {
          const float g0 = __uint_as_float(g[j]), g1 = __uint_as_float(g[j + 1]), h0 = __uint_as_float(h[j]), h1 = __uint_as_float(h[j + 1]);
          if (kDual) {
            v[0][(c + j) / 2] = pack_bf16(silu_tile(g0) * h0, silu_tile(g1) * h1);
          } else {
            v[0][(c + j) / 2] = pack_bf16(g0, g1);
            v[kTiles - 1][(c + j) / 2] = pack_bf16(h0, h1);
          }
        }
      }
      tc_fence_before();
      mbar_arrive(&acc_empty[buf]);
#pragma unroll
      for (int t = 0; t < kTiles; ++t) {
        const int f = (kDual ? wu * 128 : wu * 256 + t * 128) + quad * 32 + lane;
        if (f - lane >= p.n_features) break;                 // the second tile past an odd count
#pragma unroll
        for (int j = 0; j < kBX; j += 2) store(f, j, v[t][j / 2]);
      }
    }
    if (p.signal_flag) __threadfence_system();
  }

  tc_fence_before();
  __syncthreads();
  if (warp == 3) {
    tc_fence_after();
    tmem_dealloc(tmem, 512);
  }
  if (p.signal_flag && threadIdx.x == 0) {
    __threadfence();
    const uint32_t prev = atomicAdd(p.done_counter, 1u);
    if (prev == gridDim.x - 1) {
      *p.done_counter = 0;
      __threadfence_system();
      st_release_sys(p.signal_flag, *p.epoch);
    }
  }
}

template <bool kDual, int kBX>
static int launch_w8(const cafd_gemm_args* a, cudaStream_t stream) {
  using Cfg = W8Cfg<kBX>;
  CUtensorMap tx, tw0, tw1;
  int rc = cached_tmap_2d(&tx, a->x, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, a->x_rows_total, a->k, static_cast<uint64_t>(a->k) * 2, kBX, 64);
  if (rc) return rc;
  rc = cached_tmap_2d(&tw0, a->w0, CU_TENSOR_MAP_DATA_TYPE_UINT8, 1, a->w_rows_total, a->k, a->k, 128, kW8BK);
  if (rc) return rc;
  tw1 = tw0;
  if (kDual && (rc = cached_tmap_2d(&tw1, a->w1, CU_TENSOR_MAP_DATA_TYPE_UINT8, 1, a->w_rows_total, a->k, a->k, 128, kW8BK))) return rc;
  W8Dev p{};
  p.s0 = a->w_scale; p.s1 = a->w_scale1;
  p.out = static_cast<__nv_bfloat16*>(a->out);
  p.row_dst = a->row_dst; p.tile_expert = a->tile_expert; p.tile_row0 = a->tile_row0; p.num_x_tiles = a->num_x_tiles;
  p.wait_flag = a->wait_flag; p.epoch = a->epoch; p.done_counter = a->done_counter; p.signal_flag = a->signal_flag; p.status = a->status;
  p.nkb = a->k / kW8BK; p.n_features = a->n_features; p.ldo = a->ldo; p.w_rows_per_expert = a->w_rows_per_expert;
  p.w_units = kDual ? a->n_features / 128 : (a->n_features + 255) / 256;
  p.max_x_tiles = a->max_x_tiles;
  int dev = 0, sms = a->num_sms;
  CAFD_CHECK_CUDA(cudaGetDevice(&dev));
  if (sms <= 0) CAFD_CHECK_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
  const long long most = static_cast<long long>(p.max_x_tiles) * p.w_units;
  auto kern = gemm_w8_kernel<kDual, kBX>;
  static std::atomic<unsigned long long> set{0};               // the attribute is the device's
  const unsigned long long bit = 1ull << (dev & 63);
  if (dev > 63 || !(set.load(std::memory_order_relaxed) & bit)) {
    CAFD_CHECK_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, Cfg::kSmem));
    set.fetch_or(bit, std::memory_order_relaxed);
  }
  launch_pdl(kern, dim3(static_cast<unsigned>(most < sms ? most : sms)), dim3(kW8Threads), Cfg::kSmem, stream, tx, tw0, tw1, p);
  return static_cast<int>(cudaGetLastError());
}

}  // namespace cafd

using namespace cafd;

// Grouped product with the arguments of cafd_gemm's grouped mode: w0 (and w1: SwiGLU pair) E4M3 codes [experts * n_features, k], w_scale /
// w_scale1 a float for every 128 x 128 block, x a bf16 slab whose segments are padded to bx rows (32, 64 or 128), bf16 results.
extern "C" int cafd_gemm_w8(const cafd_gemm_args* a, cafd_stream_t stream_) {
  cudaStream_t stream = static_cast<cudaStream_t>(stream_);
  if (!a || !a->w0 || !a->x || !a->out || !a->w_scale || !a->tile_expert || !a->tile_row0 || !a->num_x_tiles || a->max_x_tiles <= 0) return -10;
  if (a->k <= 0 || a->k % kW8BK || a->n_features <= 0 || a->n_features % 128 || a->w_rows_per_expert != a->n_features || a->ldo % 2) return -10;
  if (a->dual && (!a->w1 || !a->w_scale1 || a->w1_row_offset || a->glu)) return -10;
  if (a->out_f32 || a->residual || a->row_scale || a->rs_ranks || a->n_signal_flags || a->n_wait_flags > 1) return -13;
  if ((a->signal_flag && (!a->done_counter || !a->epoch)) || (a->wait_flag && !a->epoch)) return -12;
  switch (a->bx) {
    case 32: return a->dual ? launch_w8<true, 32>(a, stream) : launch_w8<false, 32>(a, stream);
    case 64: return a->dual ? launch_w8<true, 64>(a, stream) : launch_w8<false, 64>(a, stream);
    case 128: return a->dual ? launch_w8<true, 128>(a, stream) : launch_w8<false, 128>(a, stream);
  }
  return -12;
}

CAFD_WAIT_LIMIT_SETTER(cafd_gemm_w8_set_wait_limit_ns)
