// Dense product of a decode batch (up to 128 rows, weights on the M side) whose tiles alone leave most SMs idle: the K range of a tile is cut
// over the blocks of a cluster, and their partial sums meet in shared memory.
//
// Bound by bytes in the weights, which the chain behind them hid: with partials in global memory every block waited for a fence and a ticket,
// and the last one of a tile read all of them, six round trips through L2, while the others were done.  Here each block adds its share of the
// rows from its peers' shared memory.  The cut of K and the order of the additions are those of gemm_tcgen05.cu, so the bits are the same.
// When the caller says that the previous kernel does not write the weights, the ring is filled with them before that kernel has ended.
// Behind a norm, at 17 / 32 / 64 / 128 rows (before: partials in global memory, or up to 32 rows gemm_skinny.cu): 2048 x 4096 13.1 / 17.1 /
// 23.9 / 40.0 -> 6.7 / 7.6 / 9.4 / 13.3 us, 5120 x 2048 14.1 / 15.1 / 20.9 / 33.3 -> 8.5 / 10.0 / 14.0 / 22.2, a router's 128 x 2048 6.3 /
// 8.4 / 18.6 / 32.0 -> 4.0 / 4.6 / 6.2 / 9.8, 2112 x 7168 16.6 / 17.6 / 24.4 / 38.7 -> 9.3 / 9.9 / 12.0 / 17.0 (10 rows 13.4 -> 8.9).
#include "cafd_api.h"
#include "common.cuh"
#include "host_tma.h"

#include <cooperative_groups.h>

#include <atomic>

namespace cafd {

namespace cg = cooperative_groups;

constexpr int kSplitBK = 64, kSplitThreads = 192, kSplitMax = 16;

template <int kBX>
struct SplitCfg {
  static constexpr int kWBytes = 128 * kSplitBK * 2;
  static constexpr int kStageBytes = kWBytes + kBX * kSplitBK * 2;
  static constexpr int kStages = 100 * 1024 / kStageBytes;        // two blocks per SM: clusters of nine or so need the room to be placed
  static constexpr int kSmemBytes = kStages * kStageBytes + 1024;
  static constexpr int kTmemCols = kBX < 32 ? 32 : kBX;
  static_assert(kBX * 128 * 4 <= kStages * kStageBytes, "the partial sums take the ring's place");
};

struct SplitDev {
  void* out;
  const void* residual;
  uint32_t* status;
  int num_k_blocks, n_features, x_rows, ldo, out_f32, splits, resident;
};

template <int kBX>
__global__ void __launch_bounds__(kSplitThreads, 2)
gemm_split_kernel(const __grid_constant__ CUtensorMap tm_w, const __grid_constant__ CUtensorMap tm_x, const SplitDev p) {
  using Cfg = SplitCfg<kBX>;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  __shared__ uint64_t full_bar[Cfg::kStages], empty_bar[Cfg::kStages], done_bar;
  __shared__ uint32_t tmem_slot;
  const int warp = warp_uniform(threadIdx.x >> 5), lane = threadIdx.x & 31;
  const int tile = blockIdx.x / p.splits, split = blockIdx.x - tile * p.splits;      // a cluster is a tile's splits
  const int kb0 = split * p.num_k_blocks / p.splits, n = (split + 1) * p.num_k_blocks / p.splits - kb0;
  const int ahead = p.resident ? min(n, Cfg::kStages) : 0;                           // stages whose weights do not wait for the previous kernel

  if (threadIdx.x == 0) {
    for (int s = 0; s < Cfg::kStages; ++s) {
      mbar_init(&full_bar[s], 1);
      mbar_init(&empty_bar[s], 1);
    }
    mbar_init(&done_bar, 1);
    mbar_fence_init();
    tma_prefetch_desc(&tm_w);
    tma_prefetch_desc(&tm_x);
    for (int i = 0; i < ahead; ++i) {
      mbar_expect_tx(&full_bar[i], Cfg::kStageBytes);
      tma_load_2d(smem + i * Cfg::kStageBytes, &tm_w, &full_bar[i], (kb0 + i) * kSplitBK, tile * 128);
    }
  }
  if (warp == 1) {
    tmem_alloc(&tmem_slot, Cfg::kTmemCols);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  pdl_wait();
  pdl_trigger();
  const uint32_t tmem = tmem_slot;
  float* part = reinterpret_cast<float*>(smem);                   // [row][128 features], once the ring is read

  if (warp == 0) {
    if (lane == 0) {
      for (int i = 0; i < n; ++i) {
        const int st = i % Cfg::kStages;
        if (!mbar_wait(&empty_bar[st], ((i / Cfg::kStages) & 1) ^ 1, p.status, kTimeoutEmptyBarrier)) break;
        uint8_t* w = smem + st * Cfg::kStageBytes;
        if (i >= ahead) {
          mbar_expect_tx(&full_bar[st], Cfg::kStageBytes);
          tma_load_2d(w, &tm_w, &full_bar[st], (kb0 + i) * kSplitBK, tile * 128);
        }
        tma_load_2d(w + Cfg::kWBytes, &tm_x, &full_bar[st], (kb0 + i) * kSplitBK, 0);
      }
    }
  } else if (warp == 1) {
    constexpr uint32_t idesc = make_idesc(128, kBX, 1, 1);
    const uint64_t wdesc = smem_desc_k_sw128(smem_u32(smem)), xdesc = smem_desc_k_sw128(smem_u32(smem) + Cfg::kWBytes);
    for (int i = 0; i < n; ++i) {
      const int st = i % Cfg::kStages;
      if (!mbar_wait_warp(&full_bar[st], (i / Cfg::kStages) & 1, p.status, kTimeoutFullBarrier)) break;
      tc_fence_after();
      if (elect_one()) {
        const uint64_t off = static_cast<uint64_t>(st * (Cfg::kStageBytes >> 4));
#pragma unroll
        for (int k4 = 0; k4 < kSplitBK / 16; ++k4) umma_f16(tmem, wdesc + off + k4 * 2, xdesc + off + k4 * 2, idesc, (i | k4) ? 1u : 0u);
        umma_commit(&empty_bar[st]);
        if (i == n - 1) umma_commit(&done_bar);
      }
      __syncwarp();
    }
  } else if (mbar_wait(&done_bar, 0, p.status, kTimeoutTmemFull)) {
    tc_fence_after();
    const int fl = (warp & 3) * 32 + lane;
    const uint32_t t0 = tmem + (static_cast<uint32_t>((warp & 3) * 32) << 16);
#pragma unroll 2
    for (int c0 = 0; c0 < kBX; c0 += 16) {
      if (c0 >= p.x_rows) break;
      uint32_t r[16];
      __syncwarp();
      tmem_ld_32x16(t0 + c0, r);
      tmem_ld_wait();
#pragma unroll
      for (int j = 0; j < 16; ++j) part[(c0 + j) * 128 + fl] = __uint_as_float(r[j]);
    }
    tc_fence_before();
  }
  __syncwarp();
  cg::cluster_group cluster = cg::this_cluster();
  cluster.sync();
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem, Cfg::kTmemCols);
  }
  if (warp >= 2) {                                                // thread = feature; this block's share of the rows
    const int fl = (warp - 2) * 32 + lane, f = tile * 128 + fl;
#pragma unroll 2
    for (int row = split; row < p.x_rows; row += p.splits) {
      float t[kSplitMax];
#pragma unroll
      for (int s = 0; s < kSplitMax; ++s) t[s] = s < p.splits ? cluster.map_shared_rank(part, s)[row * 128 + fl] : 0.f;
      float v = 0.f;
#pragma unroll
      for (int s = 0; s < kSplitMax; ++s)
        if (s < p.splits) v += t[s];
      if (f < p.n_features) {
        const size_t off = static_cast<size_t>(row) * p.ldo + f;
        if (p.out_f32) {
          static_cast<float*>(p.out)[off] = v;
        } else {
          if (p.residual) v += __bfloat162float(static_cast<const __nv_bfloat16*>(p.residual)[off]);
          static_cast<__nv_bfloat16*>(p.out)[off] = __float2bfloat16(v);
        }
      }
    }
  }
  cluster.sync();                                                 // the partial sums are read
}

// Blocks per tile, or 0 where gemm_tcgen05.cu's kernel takes the product: grouped, peer or flagged forms, tiles enough for the GPU, and long
// parts of many rows, which its deeper ring streams faster (7168 x 16384 in two parts at 64 / 128 rows: 62.0 / 76.1 us there, 64.3 / 84.6
// here; at 32 55.7 and 53.0).  Parts beyond a cluster's sixteen blocks are made longer.
int gemm_split_parts(const cafd_gemm_args* a) {
  if (!a->swap || a->dual || (a->bx != 16 && a->bx != 32 && a->bx != 64 && a->bx != 128) || a->x_rows > a->bx || a->tile_expert || a->tile_row0 || a->num_x_tiles || a->row_dst ||
      a->row_scale || a->rs_ranks || a->wait_flag || a->signal_flag || a->n_signal_flags || !a->splitk_scratch || !a->splitk_tickets)
    return 0;
  int sms = a->num_sms;
  if (sms <= 0) return 0;
  const int tiles = (a->n_features + 127) / 128, nkb = (a->k + kSplitBK - 1) / kSplitBK;
  long long units = a->splitk_scratch_floats / (static_cast<long long>(a->bx) * 128);
  if (units > a->splitk_ticket_count) units = a->splitk_ticket_count;
  if (tiles > units) return 0;
  long long splits = sms / tiles;
  if (splits > nkb / 4) splits = nkb / 4;
  if (splits > units / tiles) splits = units / tiles;
  if (splits < 2 || (a->bx > 32 && nkb / splits > 64)) return 0;
  return splits < kSplitMax ? static_cast<int>(splits) : kSplitMax;
}

template <int kBX>
static int launch_split(const cafd_gemm_args* a, int splits, cudaStream_t stream) {
  using Cfg = SplitCfg<kBX>;
  CUtensorMap tw, tx;
  const CUtensorMapDataType dt = CU_TENSOR_MAP_DATA_TYPE_BFLOAT16;
  const uint64_t pitch = static_cast<uint64_t>(a->k) * 2;
  int rc = cached_tmap_2d(&tw, a->w0, dt, 2, a->w_rows_total, a->k, pitch, 128, kSplitBK);
  if (rc) return rc;
  rc = cached_tmap_2d(&tx, a->x, dt, 2, a->x_rows_total, a->k, pitch, kBX, kSplitBK);
  if (rc) return rc;
  const SplitDev p{a->out, a->residual, a->status, (a->k + kSplitBK - 1) / kSplitBK, a->n_features, a->x_rows, a->ldo, a->out_f32, splits,
                   a->w_resident};
  auto kern = gemm_split_kernel<kBX>;
  static std::atomic<unsigned long long> set{0};                  // the attributes are the device's
  int dev = 0;
  CAFD_CHECK_CUDA(cudaGetDevice(&dev));
  const unsigned long long bit = 1ull << (dev & 63);
  if (dev > 63 || !(set.load(std::memory_order_relaxed) & bit)) {
    CAFD_CHECK_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, Cfg::kSmemBytes));
    CAFD_CHECK_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeNonPortableClusterSizeAllowed, 1));
    set.fetch_or(bit, std::memory_order_relaxed);
  }
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(((a->n_features + 127) / 128) * splits);
  cfg.blockDim = dim3(kSplitThreads);
  cfg.dynamicSmemBytes = Cfg::kSmemBytes;
  cfg.stream = stream;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = pdl_enabled() ? 1 : 0;
  attr[1].id = cudaLaunchAttributeClusterDimension;
  attr[1].val.clusterDim.x = splits;
  attr[1].val.clusterDim.y = attr[1].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 2;
  CAFD_CHECK_CUDA(cudaLaunchKernelEx(&cfg, kern, tw, tx, p));
  return static_cast<int>(cudaGetLastError());
}

int gemm_split(const cafd_gemm_args* a, int splits, cudaStream_t stream) {
  return a->bx == 16 ? launch_split<16>(a, splits, stream) : a->bx == 32 ? launch_split<32>(a, splits, stream) : a->bx == 64 ? launch_split<64>(a, splits, stream) : launch_split<128>(a, splits, stream);
}

}  // namespace cafd

CAFD_WAIT_LIMIT_SETTER(cafd_gemm_split_set_wait_limit_ns)
