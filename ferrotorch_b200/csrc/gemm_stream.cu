// GEMM for few rows against a large weight (decode, short prompts):  C[M, N] (+)= X[M, K] W[N, K]^T, bf16, fp32 accumulation.
//
// Such a product is bound by the bytes of W (64 rows of a 4096 x 14336 product: 117 MB, 18 us at 6.6 TB/s; 0.5 us of tensor-core time)
// and, where W is small, by the chain of latencies of one launch:
//   * W is the 128-row operand of the MMA, the rows of X are its N dimension (16 .. 256, a multiple of 16; more rows are cut into equal
//     row tiles), so that no tensor-core row is padding and X costs little shared memory;
//   * a thread-block cluster of up to eight CTAs works on one 128-row tile of W, each on its part of the contraction, so that even a
//     weight of 2048 rows is read by 128 SMs;
//   * the parts meet in shared memory: CTA j of the cluster is sent its 128 / S columns of every part, adds them in the order of the
//     contraction (the result does not depend on timing) and writes them, while the cluster's next tile is already being loaded.
//     Through a workspace in L2 the same sum took 5 us for one row and 12 us for 64 (store, fence, ticket, load);
//   * the launch overlaps the kernel before it (grid_dependency_wait), whose last microseconds bring W into L2.
// Measured, us for 1 / 64 rows, back to back in a graph, weights from HBM (before: CTA-pair tiles, pieces in a workspace and a second
// launch that adds them):     6144 x 4096     4096 x 4096    28672 x 4096   4096 x 14336   128256 x 4096   2048 x 2048    3072 x 8192
//   before                    17.5 / 18.5     15.6 / 16.6    50.3 / 53.3    28.8 / 30.5    165 / 174       11.1 / 12.0    18.7 / 19.9
//   now                       13.6 / 14.9     10.9 / 12.2    42.3 / 48.3    23.4 / 26.0    156 / 166        6.0 / 7.4     14.6 / 16.1
//   weight bytes at 6.65 TB/s  7.6             5.0           35.3           17.7           158              1.3            7.6
//
// With a gated weight [2 N, K] (gate rows, then up rows) a tile holds 64 gate rows and the 64 up rows beside them, and the results are
// act(gate) * up straight from the fp32 sums: the activation needs no pass of its own over rows that were rounded in between.
//
//   warp 0: TMA producer   warp 1: MMA issuer   warp 2: tensor memory   warps 4-11: parts and results
// Every wait is bounded.
#include "ft_host.h"
#include "gemm_flags.cuh"

namespace ft {

constexpr int ST_BM = 128, ST_BK = 64;
constexpr int ST_THREADS = 384;
constexpr int ST_EPI_WARPS = 8;
constexpr int ST_A_BYTES = ST_BM * ST_BK * 2;
constexpr int ST_BUF_BYTES = 216 * 1024;   // ring of operand tiles, then the parts that this CTA adds
constexpr int ST_MAX_STAGES = 11;
constexpr int ST_SMEM = ST_BUF_BYTES + 1024 + 512;
constexpr int ST_MAX_ROWS = 256;           // rows of X in a tile
constexpr int ST_PART_ROWS = 64;           // rows whose parts meet at a time
constexpr int ST_PARTS_BYTES = ST_BM * ST_PART_ROWS * 4;
constexpr int ST_MAX_CLUSTER = 8;
constexpr int ST_PREFETCH = 24;            // k-blocks of W that a CTA asks for while the kernel before it ends

struct StreamParams {
  void* C;
  const void* bias;
  const __nv_bfloat16* residual;
  const float *alpha, *dyt_w, *dyt_b;   // dynamic tanh of the new values (fp32 results only)
  __nv_bfloat16* dyt_out;
  float dyt_scale;
  int M, N, tiles, m_tiles, k_blocks, cluster, bn, stages, flags, accumulate, vec, vec_r;
  int n_tile;           // columns of C in a tile: 128, or 64 with a gated weight
  int glu;              // 0: none; 1 / 2 / 3: silu / relu / gelu (tanh form) of the gate
  long long ldc, ldr, ldd;
  int* status;
};

// Results (m, n .. n + 3), of which `left` exist, from their sums; bias: that of these columns.
__device__ __forceinline__ void stream_finish(const StreamParams& p, int m, int n, int left, const float (&bias)[4], float4 sum) {
  float v[4] = {sum.x + bias[0], sum.y + bias[1], sum.z + bias[2], sum.w + bias[3]};
  if (p.flags & GEMM_OUT_F32) {
    float* c = static_cast<float*>(p.C) + static_cast<long long>(m) * p.ldc + n;
    if (p.vec && left >= 4) {
      if (p.accumulate) {
        const float4 old = *reinterpret_cast<const float4*>(c);
        v[0] += old.x; v[1] += old.y; v[2] += old.z; v[3] += old.w;
      }
      *reinterpret_cast<float4*>(c) = make_float4(v[0], v[1], v[2], v[3]);
    } else {
#pragma unroll
      for (int j = 0; j < 4; ++j)
        if (j < left) {
          if (p.accumulate) v[j] += c[j];
          c[j] = v[j];
        }
    }
    if (p.dyt_out) {
      __nv_bfloat16* d = p.dyt_out + static_cast<long long>(m) * p.ldd + n;
      const float alpha = *p.alpha;
#pragma unroll
      for (int j = 0; j < 4; ++j)
        if (j < left) d[j] = __float2bfloat16((tanhf(alpha * v[j]) * p.dyt_w[n + j] + p.dyt_b[n + j]) * p.dyt_scale);
    }
    return;
  }
  if (p.residual) {
    const __nv_bfloat16* r = p.residual + static_cast<long long>(m) * p.ldr + n;
    if (p.vec_r && left >= 4) {
      const uint2 u = *reinterpret_cast<const uint2*>(r);
      const float2 a = unpack_bf16x2(u.x), b = unpack_bf16x2(u.y);
      v[0] += a.x; v[1] += a.y; v[2] += b.x; v[3] += b.y;
    } else {
#pragma unroll
      for (int j = 0; j < 4; ++j)
        if (j < left) v[j] += __bfloat162float(r[j]);
    }
  }
  if (p.flags & GEMM_ACT_MASK) {
#pragma unroll
    for (int j = 0; j < 4; ++j) v[j] = apply_act(v[j], p.flags);
  }
  __nv_bfloat16* c = static_cast<__nv_bfloat16*>(p.C) + static_cast<long long>(m) * p.ldc + n;
  if (p.vec && left >= 4) {
    *reinterpret_cast<uint2*>(c) = make_uint2(pack_bf16x2(v[0], v[1]), pack_bf16x2(v[2], v[3]));
  } else {
#pragma unroll
    for (int j = 0; j < 4; ++j)
      if (j < left) c[j] = __float2bfloat16(v[j]);
  }
}

__global__ void __launch_bounds__(ST_THREADS, 1)
gemm_stream_kernel(const __grid_constant__ CUtensorMap tmW, const __grid_constant__ CUtensorMap tmX, const StreamParams p) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~static_cast<uintptr_t>(1023));
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + ST_BUF_BYTES);
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 2 * ST_MAX_STAGES + 6);
  volatile int* abort_word = reinterpret_cast<volatile int*>(tmem_slot + 1);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t smem_base = smem_u32(smem), bar_base = smem_u32(bars);
  const int stages = p.stages, S = p.cluster;
  const int rank = static_cast<int>(cluster_ctarank());
  const uint32_t stage_bytes = ST_A_BYTES + p.bn * (ST_BK * 2);
  auto full_bar = [&](int s) { return bar_base + 8u * s; };
  auto empty_bar = [&](int s) { return bar_base + 8u * (ST_MAX_STAGES + s); };
  auto tfull_bar = [&](int a) { return bar_base + 8u * (2 * ST_MAX_STAGES + a); };
  auto tempty_bar = [&](int a) { return bar_base + 8u * (2 * ST_MAX_STAGES + 2 + a); };
  const uint32_t parts_full = bar_base + 8u * (2 * ST_MAX_STAGES + 4);   // the parts of all CTAs have arrived here
  const uint32_t parts_free = bar_base + 8u * (2 * ST_MAX_STAGES + 5);   // all CTAs have added theirs: the next parts may be sent
  const int kb0 = p.k_blocks * rank / S, kb1 = p.k_blocks * (rank + 1) / S;
  const int first = blockIdx.x / S, step = gridDim.x / S;
  uint32_t tmem_cols = 32;
  while (tmem_cols < 2u * p.bn) tmem_cols <<= 1;

  if (threadIdx.x == 0) {
    grid_dependency_launch();
    *abort_word = 0;
    for (int s = 0; s < stages; ++s) {
      mbar_init(full_bar(s), 1);
      mbar_init(empty_bar(s), 1);
    }
    for (int a = 0; a < 2; ++a) {
      mbar_init(tfull_bar(a), 1);
      mbar_init(tempty_bar(a), ST_EPI_WARPS);
    }
    mbar_init(parts_full, S * ST_EPI_WARPS);
    mbar_init(parts_free, S * ST_EPI_WARPS);
    fence_mbar_init();
    tma_prefetch_desc(&tmW);
    tma_prefetch_desc(&tmX);
    // W does not come from the kernel before this one in most uses, but it may: it is only brought into L2 ahead of the wait, and read
    // behind it
    int left = ST_PREFETCH;
    for (int tile = first; tile < p.tiles && left > 0; tile += step) {
      const int n0 = (p.m_tiles == 1 ? tile : tile / p.m_tiles) * p.n_tile;
      for (int kb = kb0; kb < kb1 && left > 0; ++kb, --left) {
        tma_prefetch_l2_2d(&tmW, kb * ST_BK, n0);
        if (p.glu) tma_prefetch_l2_2d(&tmW, kb * ST_BK, p.N + n0);
      }
    }
  }
  if (warp == 2) {
    tmem_alloc(smem_u32(tmem_slot), tmem_cols);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  cluster_sync_all();  // the peers' barriers are initialised before anything arrives on them
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  grid_dependency_wait();

  if (warp == 0) {
    // ------------------------------------------------------------------ producer
    if (lane == 0) {
      int stage = 0;
      uint32_t phase = 0;
      bool ok = true;
      for (int tile = first; tile < p.tiles && ok; tile += step) {
        const int wt = p.m_tiles == 1 ? tile : tile / p.m_tiles, n0 = wt * p.n_tile, m0 = (tile - wt * p.m_tiles) * p.bn;
        for (int kb = kb0; kb < kb1; ++kb) {
          ok = mbar_wait(empty_bar(stage), phase ^ 1u, abort_word, FT_ERR_TIMEOUT_PRODUCER);
          if (!ok) break;
          const uint32_t sW = smem_base + stage * stage_bytes;
          mbar_expect_tx(full_bar(stage), stage_bytes);
          tma_load_2d(sW, &tmW, full_bar(stage), kb * ST_BK, n0);
          if (p.glu) tma_load_2d(sW + ST_A_BYTES / 2, &tmW, full_bar(stage), kb * ST_BK, p.N + n0);
          tma_load_2d(sW + ST_A_BYTES, &tmX, full_bar(stage), kb * ST_BK, m0);
          if (++stage == stages) { stage = 0; phase ^= 1u; }
        }
      }
      if (!ok) {
        // give the loads already issued a bounded time to land before the shared memory is released
        const unsigned long long t0 = globaltimer_ns();
        while (globaltimer_ns() - t0 < 2000000ull) __nanosleep(1000);
      }
    }
  } else if (warp == 1) {
    // ------------------------------------------------------------------ MMA issuer
    if (lane == 0) {
      const uint32_t idesc = make_idesc_f16(ST_BM, p.bn, 1, 0, 0);
      int stage = 0, acc = 0;
      uint32_t phase = 0, acc_phase = 0;
      bool ok = true;
      for (int tile = first; tile < p.tiles; tile += step) {
        if (!mbar_wait(tempty_bar(acc), acc_phase ^ 1u, abort_word, FT_ERR_TIMEOUT_MMA)) break;
        tc_fence_after();
        const uint32_t d = tmem_base + static_cast<uint32_t>(acc * p.bn);
        for (int kb = kb0; kb < kb1; ++kb) {
          ok = mbar_wait(full_bar(stage), phase, abort_word, FT_ERR_TIMEOUT_MMA);
          if (!ok) break;
          tc_fence_after();
          const uint32_t sW = smem_base + stage * stage_bytes, sX = sW + ST_A_BYTES;
#pragma unroll
          for (int k = 0; k < ST_BK / 16; ++k)
            umma_f16_ss(d, make_smem_desc_sw128(sW + k * 32, 16, 1024), make_smem_desc_sw128(sX + k * 32, 16, 1024), idesc,
                        (kb > kb0 || k > 0) ? 1u : 0u);
          umma_commit(empty_bar(stage));
          if (++stage == stages) { stage = 0; phase ^= 1u; }
        }
        if (!ok) break;
        umma_commit(tfull_bar(acc));
        acc ^= 1;
        if (acc == 0) acc_phase ^= 1u;
      }
    }
  } else if (warp >= 4) {
    // ------------------------------------------------------------------ parts and results
    const int e = warp - 4, quarter = warp & 3, half = e >> 2;
    const int cols = ST_BM / S, col = quarter * 32 + lane;          // columns of C that a CTA adds; this lane's column of the tile
    const uint32_t parts = smem_base + static_cast<uint32_t>(stages) * stage_bytes;
    // Parts lie as [CTA that sent it][row of X][column]: the lanes of a warp write and read neighbouring words.  (Four rows of a column
    // as one 16-byte store to the peer took three times as long.)
    // with a gated weight a CTA adds as many gate columns as up columns, the up columns behind the others
    const int own = p.n_tile / S, gate_col = p.glu ? col & 63 : col;
    const int place = gate_col % own + (p.glu && col >= 64 ? own : 0);
    const uint32_t mine = mapa_shared(parts, gate_col / own) + static_cast<uint32_t>(rank * ST_PART_ROWS * cols + place) * 4u;
    const float* all = reinterpret_cast<const float*>(smem + stages * stage_bytes);
    const int mc = (threadIdx.x - 128) % (own / 4) * 4, mr = (threadIdx.x - 128) / (own / 4), m_step = ST_EPI_WARPS * 32 / (own / 4);
    int acc = 0;
    uint32_t acc_phase = 0, meeting = 0;
    bool ok = true;
    for (int tile = first; tile < p.tiles && ok; tile += step) {
      const int wt = p.m_tiles == 1 ? tile : tile / p.m_tiles, m0 = (tile - wt * p.m_tiles) * p.bn, rows = min(p.bn, p.M - m0);
      const int n = wt * p.n_tile + rank * own + mc, left = p.N - n;
      float bias[4] = {0.f, 0.f, 0.f, 0.f};
      if (p.flags & (GEMM_BIAS | GEMM_BIAS_F32)) {
#pragma unroll
        for (int j = 0; j < 4; ++j)
          if (j < left)
            bias[j] = (p.flags & GEMM_BIAS_F32) ? static_cast<const float*>(p.bias)[n + j]
                                                : __bfloat162float(static_cast<const __nv_bfloat16*>(p.bias)[n + j]);
      }
      ok = __all_sync(0xffffffffu, mbar_wait(tfull_bar(acc), acc_phase, abort_word, FT_ERR_TIMEOUT_EPILOGUE));
      const uint32_t t_row = tmem_base + (static_cast<uint32_t>(quarter * 32) << 16) + static_cast<uint32_t>(acc * p.bn);
      for (int r0 = 0; r0 < rows && ok; r0 += ST_PART_ROWS, ++meeting) {
        const int here = min(ST_PART_ROWS, rows - r0);
        if (meeting) ok = __all_sync(0xffffffffu, mbar_wait_cluster(parts_free, (meeting ^ 1u) & 1u, abort_word, FT_ERR_TIMEOUT_EPILOGUE));
        if (!ok) break;
        tc_fence_after();
#pragma unroll 1
        for (int c = half * 16; c < here; c += 32) {
          uint32_t r[16];
          tmem_ld_32x16(t_row + r0 + c, r);
          tmem_ld_wait();
#pragma unroll
          for (int j = 0; j < 16; ++j)
            if (c + j < here) st_cluster(mine + static_cast<uint32_t>((c + j) * cols) * 4u, r[j]);
        }
        tc_fence_before();
        __syncwarp();
        if (lane < S) mbar_arrive_cluster(mapa_shared(parts_full, lane));
        if (lane == 0 && r0 + ST_PART_ROWS >= rows) mbar_arrive(tempty_bar(acc));
        ok = __all_sync(0xffffffffu, mbar_wait_cluster(parts_full, meeting & 1u, abort_word, FT_ERR_TIMEOUT_EPILOGUE));
        if (!ok) break;
        // a thread adds four columns of every so many rows
        if (left > 0)
          for (int m = mr; m < here; m += m_step) {
            const float* src = all + m * cols + mc;
            float4 sum = *reinterpret_cast<const float4*>(src);
#pragma unroll 4
            for (int s = 1; s < S; ++s) {
              const float4 v = *reinterpret_cast<const float4*>(src + s * ST_PART_ROWS * cols);
              sum.x += v.x; sum.y += v.y; sum.z += v.z; sum.w += v.w;
            }
            if (p.glu) {
              float4 up = *reinterpret_cast<const float4*>(src + own);
#pragma unroll 4
              for (int s = 1; s < S; ++s) {
                const float4 v = *reinterpret_cast<const float4*>(src + own + s * ST_PART_ROWS * cols);
                up.x += v.x; up.y += v.y; up.z += v.z; up.w += v.w;
              }
              sum = make_float4(glu(sum.x, up.x, p.glu), glu(sum.y, up.y, p.glu), glu(sum.z, up.z, p.glu),
                                glu(sum.w, up.w, p.glu));
            }
            stream_finish(p, m0 + r0 + m, n, left, bias, sum);
          }
        __syncwarp();
        if (lane < S) mbar_arrive_cluster(mapa_shared(parts_free, lane));
      }
      acc ^= 1;
      if (acc == 0) acc_phase ^= 1u;
    }
  }

  tc_fence_before();
  __syncthreads();
  cluster_sync_all();  // no CTA leaves while a peer can still reach its shared memory
  if (warp == 2) {
    tc_fence_after();
    tmem_dealloc(tmem_base, tmem_cols);
  }
  if (threadIdx.x == 0 && *abort_word != 0 && p.status != nullptr) atomicCAS(p.status, 0, *abort_word);
}

static int launch_stream(const void* X, const void* W, StreamParams p, int K, long long ldx, long long ldw, int device, cudaStream_t stream) {
  static std::atomic<int> known_clusters[64][4];
  int max_clusters[4];
  if (int rc = resident_clusters(known_clusters, gemm_stream_kernel, ST_THREADS, ST_SMEM, device, max_clusters)) return rc;
  p.m_tiles = (p.M + ST_MAX_ROWS - 1) / ST_MAX_ROWS;
  p.bn = ((p.M + p.m_tiles - 1) / p.m_tiles + 15) / 16 * 16;
  p.m_tiles = (p.M + p.bn - 1) / p.bn;
  p.stages = (ST_BUF_BYTES - ST_PARTS_BYTES) / (ST_A_BYTES + p.bn * ST_BK * 2);
  if (p.stages > ST_MAX_STAGES) p.stages = ST_MAX_STAGES;
  p.k_blocks = (K + ST_BK - 1) / ST_BK;
  p.n_tile = p.glu ? ST_BM / 2 : ST_BM;
  p.tiles = (p.N + p.n_tile - 1) / p.n_tile * p.m_tiles;
  p.status = device_status_word(device);
  cudaLaunchAttribute attr[2] = {};
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
  attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[1].val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t cfg{};
  cfg.blockDim = ST_THREADS; cfg.dynamicSmemBytes = ST_SMEM; cfg.stream = stream; cfg.attrs = attr; cfg.numAttrs = 2;
  // CTAs per tile, as measured with clusters of 1 / 2 / 4 / 8 (us, one row): two where there are tiles enough for that (128256 x 4096:
  // 163 / 156 / 169 / 245; 28672 x 4096: 46 / 42 / 43 / 57; 16384 x 2048: 17 / 16 / 17 / 26), else four (6144 x 4096: 24 / 16 / 14 / 15;
  // 4096 x 14336: 67 / 38 / 24 / 28; 3072 x 3072: 17 / 11 / 9 / 9), and eight for a few tiles with a long contraction (2048 x 8192:
  // 41 / 22 / 14 / 13; 3072 x 8192: 40 / 24 / 16 / 15).
  int lg = p.tiles > 64 ? 1 : (p.tiles <= 24 && p.k_blocks >= 128 ? 3 : 2);
  while ((1 << lg) > p.k_blocks) --lg;
  p.cluster = 1 << lg;
  attr[0].val.clusterDim.x = p.cluster;
  cfg.gridDim = (p.tiles < max_clusters[lg] ? p.tiles : max_clusters[lg]) * p.cluster;
  CUtensorMap tmW, tmX;
  int rc = make_tmap_2d(&tmW, W, 2, K, p.glu ? 2ull * p.N : p.N, ldw * 2, ST_BK, p.n_tile, 3);
  if (rc) return rc;
  rc = make_tmap_2d(&tmX, X, 2, K, p.M, ldx * 2, ST_BK, p.bn, 3);
  if (rc) return rc;
  FT_CUDA_CHECK(cudaLaunchKernelEx(&cfg, gemm_stream_kernel, tmW, tmX, p));
  count_launch();
  return FT_E_OK;
}

static bool aligned(const void* p, int bytes) { return (reinterpret_cast<uintptr_t>(p) & (bytes - 1)) == 0; }

}  // namespace ft

// C[M, N] = act(X[M, K] W[N, K]^T (+ bias[N]) (+ residual[M, N])), all bf16, K-major, strides in elements; any number of rows.
FT_API int ft_gemm_stream(const void* X, const void* W, void* C, const void* bias, const void* residual, int M, int N, int K,
                          long long ldx, long long ldw, long long ldc, long long ldr, int flags, int device, cudaStream_t stream) {
  if (int _rc = ft::ensure_device(device)) return _rc;
  using namespace ft;
  FT_REQUIRE(X && W && C, "ft_gemm_stream: null operand");
  FT_REQUIRE(M > 0 && N > 0 && K > 0, "ft_gemm_stream: empty problem %dx%dx%d", M, N, K);
  FT_REQUIRE(ldx % 8 == 0 && ldw % 8 == 0 && N % 8 == 0, "ft_gemm_stream: strides and N must be multiples of 8");
  FT_REQUIRE(!(flags & (GEMM_OUT_F32 | GEMM_ACCUMULATE)), "ft_gemm_stream: bf16 output, no accumulation");
  FT_REQUIRE(!(flags & (GEMM_BIAS | GEMM_BIAS_F32)) || bias, "ft_gemm_stream: bias flag without bias");
  StreamParams p{};
  p.C = C; p.bias = bias; p.residual = static_cast<const __nv_bfloat16*>(residual);
  p.M = M; p.N = N; p.flags = flags & 0xFFFF; p.ldc = ldc; p.ldr = ldr;
  p.vec = ldc % 4 == 0 && aligned(C, 8);
  p.vec_r = ldr % 4 == 0 && aligned(residual, 8);
  return launch_stream(X, W, p, K, ldx, ldw, device, stream);
}

// C[M, F] = act(gate) * up of X [M, K] with a gated weight W [2 F, K] (gate rows, then up rows); act: 0 silu, 1 relu, 2 gelu (tanh form).
FT_API int ft_gemm_stream_glu(const void* X, const void* W, void* C, int M, int F, int K, long long ldx, long long ldw, long long ldc, int act,
                              int device, cudaStream_t stream) {
  if (int _rc = ft::ensure_device(device)) return _rc;
  using namespace ft;
  FT_REQUIRE(X && W && C, "ft_gemm_stream_glu: null operand");
  FT_REQUIRE(M > 0 && F > 0 && K > 0 && act >= 0 && act <= 2, "ft_gemm_stream_glu: bad problem %dx%dx%d", M, F, K);
  FT_REQUIRE(ldx % 8 == 0 && ldw % 8 == 0 && F % 8 == 0, "ft_gemm_stream_glu: strides and F must be multiples of 8");
  StreamParams p{};
  p.C = C; p.M = M; p.N = F; p.glu = act + 1; p.ldc = ldc;
  p.vec = ldc % 4 == 0 && aligned(C, 8);
  return launch_stream(X, W, p, K, ldx, ldw, device, stream);
}

// The same for a small batch M <= 128 (decode).
FT_API int ft_gemm_small_m(const void* X, const void* W, void* C, const void* bias, const void* residual, int M, int N, int K,
                           long long ldx, long long ldw, long long ldc, long long ldr, int flags, int device, cudaStream_t stream) {
  using namespace ft;
  FT_REQUIRE(M > 0 && M <= 128 && N > 0 && K > 0, "ft_gemm_small_m: M=%d must be in 1..128 (N=%d K=%d)", M, N, K);
  return ft_gemm_stream(X, W, C, bias, residual, M, N, K, ldx, ldw, ldc, ldr, flags, device, stream);
}

// C[M, N] (fp32) (+)= X[M, K] W[N, K]^T for a small batch M <= 128; with dyt_out also the next layer's dynamic tanh of the new values,
// dyt_out[M, N] = (tanh(alpha C) w + b) * dyt_scale as bf16 (being element by element, that norm needs no pass of its own over the
// residual stream).
FT_API int ft_gemm_small_m_f32(const void* X, const void* W, float* C, int accumulate, const float* alpha, const float* dyt_w,
                               const float* dyt_b, void* dyt_out, float dyt_scale, int M, int N, int K, long long ldx,
                               long long ldw, long long ldc, long long ldd, int device, cudaStream_t stream) {
  if (int _rc = ft::ensure_device(device)) return _rc;
  using namespace ft;
  FT_REQUIRE(X && W && C, "ft_gemm_small_m_f32: null operand");
  FT_REQUIRE(M > 0 && M <= 128 && N > 0 && K > ST_BK, "ft_gemm_small_m_f32: M=%d must be in 1..128, K=%d above %d (N=%d)", M, K, ST_BK, N);
  FT_REQUIRE(ldx % 8 == 0 && ldw % 8 == 0, "ft_gemm_small_m_f32: strides must be multiples of 8");
  FT_REQUIRE(!dyt_out || (alpha && dyt_w && dyt_b), "ft_gemm_small_m_f32: the fused norm needs its parameters");
  StreamParams p{};
  p.C = C; p.M = M; p.N = N; p.flags = GEMM_OUT_F32; p.accumulate = accumulate; p.ldc = ldc;
  p.alpha = alpha; p.dyt_w = dyt_w; p.dyt_b = dyt_b; p.dyt_out = static_cast<__nv_bfloat16*>(dyt_out); p.dyt_scale = dyt_scale; p.ldd = ldd;
  p.vec = ldc % 4 == 0 && aligned(C, 16);
  return launch_stream(X, W, p, K, ldx, ldw, device, stream);
}
