// Products with GGUF Q4_0 weights:  Y[M, N] = X[M, K] dequant(W)[N, K]^T (+ bias[N]), X bf16, fp32 accumulation.
//
// W stays 4-bit in HBM (32-element blocks: fp16 scale d and 16 bytes; element j = low nibble of byte j, element j + 16 = high nibble,
// value (q - 8) d, the GGML file format's order; the reference's decoder emits the nibbles of byte j as elements 2j, 2j + 1 instead,
// ferrotorch-serialize/src/gguf.rs:543-577; data in that convention is re-packed on the host, csrc/host/gguf.cpp ftg_repack_nibbles).
// The reference dequantises the whole tensor to f32 on the GPU, bounces it through the host and stores bf16
// (ferrotorch-llama/src/gpu_gguf.rs:14-27); it has no fused product.
//
// For few rows such a product is bound by expanding W: 28672 x 8192 weights are 132 MB (20 us at 6.6 TB/s), but at 2.4 instructions
// each 15 us of every SM's issue slots, so:
//   * W is the 128-row operand of the MMA and is expanded once whatever M <= 256 is; X is its N dimension;
//   * eight warps expand: a thread owns a row, turns 32 bytes into 64 bf16 with byte permutes and packed bf16 arithmetic, and writes
//     them to tensor memory, from where the MMA takes its A operand; no swizzled shared-memory tile, no proxy fence;
//   * the value is exact before its one rounding to bf16: q - 8 has 4 bits, d is split into its upper 8 bits and the 3 below them, so
//     (q - 8) d_lo is exact and the fused multiply-add (q - 8) d_hi + that rounds once: the same bits as an fp32 product would give;
//   * clusters share the contraction of a tile and meet in shared memory, as in gemm_stream.cu.
// Measured, 32 x 28672 x 8192: 103 us, 126 us when W was expanded in fp32 into a shared-memory tile, by 128 x 128 tiles of M and N.
// It stays far from both figures: issue slots are 40 % busy, HBM 15 %.  Twelve expanding warps, scales through the ring and sixteen k-blocks
// of X in flight change nothing (103 us); expanded tiles in shared memory cost more (107).
//
//   warp 0: TMA (X)   warp 1: MMA   warp 2: tensor memory   warp 3: TMA (W)   warps 4-11: expansion   warps 12-15: parts and results
// Every wait is bounded.
#include "ft_host.h"
#include "ft_ptx.cuh"

namespace ft {

constexpr int Q4_BM = 128, Q4_BK = 64, Q4_CK = 4;      // k-blocks in a block of compressed bytes (128 bytes of a row)
constexpr int Q4_THREADS = 512;
constexpr int Q4_EXPANDERS = 8;                        // warps
constexpr int Q4_COMP_BYTES = Q4_BM * 128;
constexpr int Q4_A_BUFS = 8, Q4_A_COLS = Q4_BK / 2;    // expanded k-blocks in tensor memory
constexpr int Q4_PART_ROWS = 64;                       // rows of X whose parts meet at a time
constexpr int Q4_PARTS_BYTES = Q4_BM * Q4_PART_ROWS * 4;
constexpr int Q4_MAX_STAGES = 8;
constexpr int Q4_BUF_BYTES = 220 * 1024;
constexpr int Q4_SMEM = Q4_BUF_BYTES + 1024 + 512;
constexpr int Q4_MAX_ROWS = 256;

struct Q4Params {
  void* C;
  const __nv_bfloat16* bias;
  const uint8_t* scales;
  int M, N, K, tiles, m_tiles, c_blocks, cluster, bn, accs, x_stages, c_stages, out_f32, vec;
  long long ldc;
  int* status;
};

// Upper 8 bits of an fp16 scale and the rest, each exact as bf16, in both halves of a word.
__device__ __forceinline__ void q4_scale(uint32_t half_bits, __nv_bfloat162& hi, __nv_bfloat162& lo) {
  const float d = __half2float(__ushort_as_half(static_cast<unsigned short>(half_bits)));
  float top = __uint_as_float(__float_as_uint(d) & 0xFFFF0000u), rest = d - top;
  if (!(fabsf(d) <= 65504.f)) { top = d; rest = 0.f; }             // infinity and NaN stay what they are
  hi = __float2bfloat162_rn(top);
  lo = __float2bfloat162_rn(rest);
}

// Four weights of a word of low nibbles as two bf16 pairs: 0x4300 | q is 128 + q.
__device__ __forceinline__ void q4_expand4(uint32_t nibbles, __nv_bfloat162 hi, __nv_bfloat162 lo, uint32_t& a, uint32_t& b) {
  const __nv_bfloat162 bias = __float2bfloat162_rn(-136.f);
  const uint32_t w[2] = {__byte_perm(nibbles, 0x43434343u, 0x4140), __byte_perm(nibbles, 0x43434343u, 0x4342)};
  uint32_t o[2];
#pragma unroll
  for (int i = 0; i < 2; ++i) {
    const __nv_bfloat162 q = __hadd2_rn(*reinterpret_cast<const __nv_bfloat162*>(&w[i]), bias);
    const __nv_bfloat162 v = __hfma2(q, hi, __hmul2_rn(q, lo));
    o[i] = *reinterpret_cast<const uint32_t*>(&v);
  }
  a = o[0];
  b = o[1];
}

// A block of 32 weights (16 bytes) as 16 words of pairs in the order of the contraction.
__device__ __forceinline__ void q4_expand_block(const uint4& q, uint32_t scale, uint32_t* out) {
  __nv_bfloat162 hi, lo;
  q4_scale(scale, hi, lo);
  const uint32_t w[4] = {q.x, q.y, q.z, q.w};
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    q4_expand4(w[i] & 0x0F0F0F0Fu, hi, lo, out[2 * i], out[2 * i + 1]);
    q4_expand4((w[i] >> 4) & 0x0F0F0F0Fu, hi, lo, out[8 + 2 * i], out[8 + 2 * i + 1]);
  }
}

__device__ __forceinline__ void q4_finish(const Q4Params& p, int m, int n, int left, const float (&bias)[4], float4 sum) {
  const float v[4] = {sum.x + bias[0], sum.y + bias[1], sum.z + bias[2], sum.w + bias[3]};
  const long long at = static_cast<long long>(m) * p.ldc + n;
  if (p.out_f32) {
    float* c = static_cast<float*>(p.C) + at;
    if (p.vec && left >= 4) {
      *reinterpret_cast<float4*>(c) = make_float4(v[0], v[1], v[2], v[3]);
    } else {
#pragma unroll
      for (int j = 0; j < 4; ++j)
        if (j < left) c[j] = v[j];
    }
    return;
  }
  __nv_bfloat16* c = static_cast<__nv_bfloat16*>(p.C) + at;
  if (p.vec && left >= 4) {
    *reinterpret_cast<uint2*>(c) = make_uint2(pack_bf16x2(v[0], v[1]), pack_bf16x2(v[2], v[3]));
  } else {
#pragma unroll
    for (int j = 0; j < 4; ++j)
      if (j < left) c[j] = __float2bfloat16(v[j]);
  }
}

__global__ void __launch_bounds__(Q4_THREADS, 1)
q4_gemm_kernel(const __grid_constant__ CUtensorMap tmW, const __grid_constant__ CUtensorMap tmX, const Q4Params p) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~static_cast<uintptr_t>(1023));
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + Q4_BUF_BYTES);
  enum { X_FULL = 0, X_EMPTY = X_FULL + Q4_MAX_STAGES, C_FULL = X_EMPTY + Q4_MAX_STAGES, C_EMPTY = C_FULL + Q4_MAX_STAGES,
         A_FULL = C_EMPTY + Q4_MAX_STAGES, A_EMPTY = A_FULL + Q4_A_BUFS, D_FULL = A_EMPTY + Q4_A_BUFS, D_EMPTY = D_FULL + 2,
         PARTS_FULL = D_EMPTY + 2, PARTS_FREE, NBARS };
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + NBARS);
  volatile int* abort_word = reinterpret_cast<volatile int*>(tmem_slot + 1);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t smem_base = smem_u32(smem), bar_base = smem_u32(bars);
  auto bar = [&](int i) { return bar_base + 8u * i; };
  const int S = p.cluster, rank = static_cast<int>(cluster_ctarank());
  const uint32_t x_bytes = p.bn * (Q4_BK * 2);
  const uint32_t comp_base = smem_base + p.x_stages * x_bytes;
  const uint32_t parts_off = p.x_stages * x_bytes + p.c_stages * Q4_COMP_BYTES;
  const int k_blocks = (p.K + Q4_BK - 1) / Q4_BK;
  const int cb0 = p.c_blocks * rank / S, cb1 = p.c_blocks * (rank + 1) / S;      // this CTA's part of a contraction
  const int kb0 = cb0 * Q4_CK, kb1 = min(cb1 * Q4_CK, k_blocks);
  const int first = blockIdx.x / S, step = gridDim.x / S;

  if (threadIdx.x == 0) {
    grid_dependency_launch();
    *abort_word = 0;
    for (int s = 0; s < Q4_MAX_STAGES; ++s) {
      mbar_init(bar(X_FULL + s), 1);
      mbar_init(bar(X_EMPTY + s), 1);
      mbar_init(bar(C_FULL + s), 1);
      mbar_init(bar(C_EMPTY + s), Q4_EXPANDERS);
    }
    for (int s = 0; s < Q4_A_BUFS; ++s) {
      mbar_init(bar(A_FULL + s), 4);
      mbar_init(bar(A_EMPTY + s), 1);
    }
    for (int a = 0; a < 2; ++a) {
      mbar_init(bar(D_FULL + a), 1);
      mbar_init(bar(D_EMPTY + a), 4);
    }
    mbar_init(bar(PARTS_FULL), S * 4);
    mbar_init(bar(PARTS_FREE), S * 4);
    fence_mbar_init();
    tma_prefetch_desc(&tmW);
    tma_prefetch_desc(&tmX);
    int left = 12;      // a hint ahead of the wait, as in gemm_stream.cu
    for (int tile = first; tile < p.tiles && left > 0; tile += step)
      for (int cb = cb0; cb < cb1 && left > 0; ++cb, --left) tma_prefetch_l2_2d(&tmW, cb * 128, tile / p.m_tiles * Q4_BM);
  }
  if (warp == 2) {
    tmem_alloc(smem_u32(tmem_slot), 512);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  cluster_sync_all();  // the peers' barriers are initialised before anything arrives on them
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  const uint32_t tmem_a = tmem_base + 256u;                     // accumulators: columns 0 .. 255
  grid_dependency_wait();

  if (warp == 0) {
    // ------------------------------------------------------------------ X
    if (lane == 0) {
      int stage = 0;
      uint32_t phase = 0;
      bool ok = true;
      for (int tile = first; tile < p.tiles && ok; tile += step)
        for (int kb = kb0; kb < kb1; ++kb) {
          ok = mbar_wait(bar(X_EMPTY + stage), phase ^ 1u, abort_word, FT_ERR_TIMEOUT_PRODUCER);
          if (!ok) break;
          mbar_expect_tx(bar(X_FULL + stage), x_bytes);
          tma_load_2d(smem_base + stage * x_bytes, &tmX, bar(X_FULL + stage), kb * Q4_BK, tile % p.m_tiles * p.bn);
          if (++stage == p.x_stages) { stage = 0; phase ^= 1u; }
        }
      if (!ok) { const unsigned long long t0 = globaltimer_ns(); while (globaltimer_ns() - t0 < 2000000ull) __nanosleep(1000); }
    }
  } else if (warp == 3) {
    // ------------------------------------------------------------------ compressed rows of W
    if (lane == 0) {
      int stage = 0;
      uint32_t phase = 0;
      bool ok = true;
      for (int tile = first; tile < p.tiles && ok; tile += step)
        for (int cb = cb0; cb < cb1; ++cb) {
          ok = mbar_wait(bar(C_EMPTY + stage), phase ^ 1u, abort_word, FT_ERR_TIMEOUT_PRODUCER);
          if (!ok) break;
          mbar_expect_tx(bar(C_FULL + stage), Q4_COMP_BYTES);
          tma_load_2d(comp_base + stage * Q4_COMP_BYTES, &tmW, bar(C_FULL + stage), cb * 128, tile / p.m_tiles * Q4_BM);
          if (++stage == p.c_stages) { stage = 0; phase ^= 1u; }
        }
      if (!ok) { const unsigned long long t0 = globaltimer_ns(); while (globaltimer_ns() - t0 < 2000000ull) __nanosleep(1000); }
    }
  } else if (warp == 1) {
    // ------------------------------------------------------------------ MMA
    if (lane == 0) {
      const uint32_t idesc = make_idesc_f16(Q4_BM, p.bn, 1, 0, 0);
      int stage = 0, buf = 0, acc = 0;
      uint32_t phase = 0, a_phase = 0, d_phase = 0;
      bool ok = true;
      for (int tile = first; tile < p.tiles; tile += step) {
        if (!mbar_wait(bar(D_EMPTY + acc), d_phase ^ 1u, abort_word, FT_ERR_TIMEOUT_MMA)) break;
        tc_fence_after();
        const uint32_t d = tmem_base + static_cast<uint32_t>(acc * 128);
        for (int kb = kb0; kb < kb1; ++kb) {
          ok = mbar_wait(bar(X_FULL + stage), phase, abort_word, FT_ERR_TIMEOUT_MMA) &&
               mbar_wait(bar(A_FULL + buf), a_phase, abort_word, FT_ERR_TIMEOUT_MMA);
          if (!ok) break;
          tc_fence_after();
          const uint32_t sX = smem_base + stage * x_bytes, a = tmem_a + static_cast<uint32_t>(buf * Q4_A_COLS);
#pragma unroll
          for (int k = 0; k < Q4_BK / 16; ++k)
            umma_f16_ts(d, a + k * 8, make_smem_desc_sw128(sX + k * 32, 16, 1024), idesc, (kb > kb0 || k > 0) ? 1u : 0u);
          umma_commit(bar(X_EMPTY + stage));
          umma_commit(bar(A_EMPTY + buf));
          if (++stage == p.x_stages) { stage = 0; phase ^= 1u; }
          if (++buf == Q4_A_BUFS) { buf = 0; a_phase ^= 1u; }
        }
        if (!ok) break;
        umma_commit(bar(D_FULL + acc));
        if (++acc == p.accs) { acc = 0; d_phase ^= 1u; }
      }
    }
  } else if (warp >= 4 && warp < 12) {
    // ------------------------------------------------------------------ expansion
    // Two groups of four warps take every second k-block; thread r of a group owns row r of the tile.
    const int grp = (warp - 4) >> 2, quarter = warp & 3, r = quarter * 32 + lane;
    const uint32_t lane_addr = tmem_a + (static_cast<uint32_t>(quarter * 32) << 16);
    const long long scale_row = p.K >> 4;                       // bytes
    int stage = 0;
    uint32_t phase = 0;
    uint32_t done = 0;                                          // k-blocks of the CTA before this block: where it lies in the ring
    bool ok = true;
    for (int tile = first; tile < p.tiles && ok; tile += step) {
      const int n = tile / p.m_tiles * Q4_BM + r;
      const uint8_t* srow = p.scales + static_cast<long long>(min(n, p.N - 1)) * scale_row;
      // the two scales of each of a block's four k-blocks; loaded a block ahead
      auto load_scales = [&](int cb, uint32_t (&s)[Q4_CK]) {
#pragma unroll
        for (int j = 0; j < Q4_CK; ++j)
          s[j] = cb < cb1 && cb * Q4_CK + j < k_blocks ? *reinterpret_cast<const uint32_t*>(srow + (cb * Q4_CK + j) * 4) : 0u;
      };
      uint32_t next[Q4_CK];
      load_scales(cb0, next);
      for (int cb = cb0; cb < cb1 && ok; ++cb) {
        uint32_t sc[Q4_CK];
#pragma unroll
        for (int j = 0; j < Q4_CK; ++j) sc[j] = next[j];
        load_scales(cb + 1, next);
        ok = __all_sync(0xffffffffu, mbar_wait(bar(C_FULL + stage), phase, abort_word, FT_ERR_TIMEOUT_PRODUCER));
        const uint32_t row = comp_base + stage * Q4_COMP_BYTES + r * 128;
        const int count = min(Q4_CK, kb1 - cb * Q4_CK);
#pragma unroll
        for (int j = 0; j < Q4_CK; ++j) {
          if (j >= count || !ok || ((done + j) & 1u) != static_cast<uint32_t>(grp)) continue;
          uint4 q[2];
#pragma unroll
          for (int h = 0; h < 2; ++h)
            asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];"
                         : "=r"(q[h].x), "=r"(q[h].y), "=r"(q[h].z), "=r"(q[h].w)
                         : "r"(row + (static_cast<uint32_t>((2 * j + h) ^ (r & 7)) << 4)) : "memory");
          uint32_t out[32];
          q4_expand_block(q[0], sc[j] & 0xFFFFu, out);
          q4_expand_block(q[1], sc[j] >> 16, out + 16);
          const uint32_t at = done + j, buf = at % Q4_A_BUFS;
          ok = __all_sync(0xffffffffu, mbar_wait(bar(A_EMPTY + buf), ((at / Q4_A_BUFS) & 1u) ^ 1u, abort_word, FT_ERR_TIMEOUT_PRODUCER));
          if (!ok) continue;
          tc_fence_after();
          tmem_st_32x32(lane_addr + buf * Q4_A_COLS, out);
          tmem_st_wait();
          tc_fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive(bar(A_FULL + buf));
        }
        done += count;
        __syncwarp();
        if (lane == 0) mbar_arrive(bar(C_EMPTY + stage));
        if (++stage == p.c_stages) { stage = 0; phase ^= 1u; }
      }
    }
  } else if (warp >= 12) {
    // ------------------------------------------------------------------ parts and results (see gemm_stream.cu)
    const int quarter = warp & 3, tid = threadIdx.x - 384;
    const int cols = Q4_BM / S, col = quarter * 32 + lane;
    const uint32_t mine = mapa_shared(smem_base + parts_off, col / cols) + static_cast<uint32_t>(rank * Q4_PART_ROWS * cols + col % cols) * 4u;
    const float* all = reinterpret_cast<const float*>(smem + parts_off);
    const int mc = tid % (cols / 4) * 4, mr = tid / (cols / 4), m_step = 128 / (cols / 4);
    int acc = 0;
    uint32_t d_phase = 0, meeting = 0;
    bool ok = true;
    for (int tile = first; tile < p.tiles && ok; tile += step) {
      const int m0 = tile % p.m_tiles * p.bn, rows = min(p.bn, p.M - m0);
      const int n = tile / p.m_tiles * Q4_BM + rank * cols + mc, left = p.N - n;
      float bias[4] = {0.f, 0.f, 0.f, 0.f};
      if (p.bias) {
#pragma unroll
        for (int j = 0; j < 4; ++j)
          if (j < left) bias[j] = __bfloat162float(p.bias[n + j]);
      }
      ok = __all_sync(0xffffffffu, mbar_wait(bar(D_FULL + acc), d_phase, abort_word, FT_ERR_TIMEOUT_EPILOGUE));
      const uint32_t t_row = tmem_base + (static_cast<uint32_t>(quarter * 32) << 16) + static_cast<uint32_t>(acc * 128);
      for (int r0 = 0; r0 < rows && ok; r0 += Q4_PART_ROWS, ++meeting) {
        const int here = min(Q4_PART_ROWS, rows - r0);
        if (meeting) ok = __all_sync(0xffffffffu, mbar_wait_cluster(bar(PARTS_FREE), (meeting ^ 1u) & 1u, abort_word, FT_ERR_TIMEOUT_EPILOGUE));
        if (!ok) break;
        tc_fence_after();
#pragma unroll 1
        for (int c = 0; c < here; c += 16) {
          uint32_t v[16];
          tmem_ld_32x16(t_row + r0 + c, v);
          tmem_ld_wait();
#pragma unroll
          for (int j = 0; j < 16; ++j)
            if (c + j < here) st_cluster(mine + static_cast<uint32_t>((c + j) * cols) * 4u, v[j]);
        }
        tc_fence_before();
        __syncwarp();
        if (lane < S) mbar_arrive_cluster(mapa_shared(bar(PARTS_FULL), lane));
        if (lane == 0 && r0 + Q4_PART_ROWS >= rows) mbar_arrive(bar(D_EMPTY + acc));
        ok = __all_sync(0xffffffffu, mbar_wait_cluster(bar(PARTS_FULL), meeting & 1u, abort_word, FT_ERR_TIMEOUT_EPILOGUE));
        if (!ok) break;
        if (left > 0)
          for (int m = mr; m < here; m += m_step) {
            const float* src = all + m * cols + mc;
            float4 sum = *reinterpret_cast<const float4*>(src);
#pragma unroll 4
            for (int s = 1; s < S; ++s) {
              const float4 v = *reinterpret_cast<const float4*>(src + s * Q4_PART_ROWS * cols);
              sum.x += v.x; sum.y += v.y; sum.z += v.z; sum.w += v.w;
            }
            q4_finish(p, m0 + r0 + m, n, left, bias, sum);
          }
        __syncwarp();
        if (lane < S) mbar_arrive_cluster(mapa_shared(bar(PARTS_FREE), lane));
      }
      if (++acc == p.accs) { acc = 0; d_phase ^= 1u; }
    }
  }

  tc_fence_before();
  __syncthreads();
  cluster_sync_all();  // no CTA leaves while a peer can still reach its shared memory
  if (warp == 2) {
    tc_fence_after();
    tmem_dealloc(tmem_base, 512);
  }
  if (threadIdx.x == 0 && *abort_word != 0 && p.status != nullptr) atomicCAS(p.status, 0, *abort_word);
}

}  // namespace ft

// y[M,N] = x[M,K] (bf16, row stride ldx) * dequant_q4_0(nibbles [N, K/2], scales fp16 [N, K/32])^T (+ bias, bf16).
FT_API int ft_q4_0_gemm(const void* x, const void* nibbles, const void* scales, void* y, const void* bias, int M,
                        int N, int K, long long ldx, long long ldy, int out_f32, int device, cudaStream_t stream) {
  if (int _rc = ft::ensure_device(device)) return _rc;
  using namespace ft;
  FT_REQUIRE(x && nibbles && scales && y, "ft_q4_0_gemm: null pointer");
  FT_REQUIRE(M > 0 && N > 0 && K > 0 && K % 64 == 0 && N % 8 == 0 && ldx % 8 == 0 && ldy % (out_f32 ? 4 : 8) == 0,
             "ft_q4_0_gemm: K must be a multiple of 64, N of 8");
  FT_REQUIRE((reinterpret_cast<uintptr_t>(nibbles) & 15) == 0 && (reinterpret_cast<uintptr_t>(scales) & 3) == 0,
             "ft_q4_0_gemm: nibble plane must be 16-byte aligned");
  static std::atomic<int> known_clusters[64][4];
  int max_clusters[4];
  if (int rc = resident_clusters(known_clusters, q4_gemm_kernel, Q4_THREADS, Q4_SMEM, device, max_clusters)) return rc;
  Q4Params p{};
  p.C = y; p.bias = static_cast<const __nv_bfloat16*>(bias); p.scales = static_cast<const uint8_t*>(scales);
  p.M = M; p.N = N; p.K = K; p.out_f32 = out_f32; p.ldc = ldy;
  p.vec = (reinterpret_cast<uintptr_t>(y) & (out_f32 ? 15 : 7)) == 0;
  p.m_tiles = (M + Q4_MAX_ROWS - 1) / Q4_MAX_ROWS;
  p.bn = ((M + p.m_tiles - 1) / p.m_tiles + 15) / 16 * 16;
  p.m_tiles = (M + p.bn - 1) / p.bn;
  p.accs = p.bn <= 128 ? 2 : 1;
  // the compressed rows keep HBM busy, X comes from L2
  p.x_stages = p.bn <= 128 ? 4 : 3;
  p.c_stages = (Q4_BUF_BYTES - Q4_PARTS_BYTES - p.x_stages * p.bn * Q4_BK * 2) / Q4_COMP_BYTES;
  if (p.c_stages > Q4_MAX_STAGES) p.c_stages = Q4_MAX_STAGES;
  p.c_blocks = (K + Q4_BK * Q4_CK - 1) / (Q4_BK * Q4_CK);
  p.tiles = (N + Q4_BM - 1) / Q4_BM * p.m_tiles;
  p.status = device_status_word(device);
  cudaLaunchAttribute attr[2] = {};
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
  attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[1].val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t cfg{};
  cfg.blockDim = Q4_THREADS; cfg.dynamicSmemBytes = Q4_SMEM; cfg.stream = stream; cfg.attrs = attr; cfg.numAttrs = 2;
  // Bound by expansion, so the SMs have to be equally busy: the cluster size with the fewest compressed blocks in a row (rounds of
  // tiles times a CTA's part of a contraction; a part below two blocks gains nothing).  Ties go to the smaller cluster.
  int lg = 0;
  long long best = 0;
  for (int i = 0; i <= 3 && (1 << i) <= p.c_blocks; ++i) {
    const int rounds = (p.tiles + max_clusters[i] - 1) / max_clusters[i], part = (p.c_blocks + (1 << i) - 1) >> i;
    const long long cost = static_cast<long long>(rounds) * (part > 2 ? part : 2);
    if (i == 0 || cost < best) { best = cost; lg = i; }
  }
  p.cluster = 1 << lg;
  attr[0].val.clusterDim.x = p.cluster;
  cfg.gridDim = (p.tiles < max_clusters[lg] ? p.tiles : max_clusters[lg]) * p.cluster;
  CUtensorMap tmW, tmX;
  int rc = make_tmap_2d(&tmW, nibbles, 1, K / 2, N, K / 2, 128, Q4_BM, 3);
  if (rc) return rc;
  rc = make_tmap_2d(&tmX, x, 2, K, M, ldx * 2, Q4_BK, p.bn, 3);
  if (rc) return rc;
  FT_CUDA_CHECK(cudaLaunchKernelEx(&cfg, q4_gemm_kernel, tmW, tmX, p));
  count_launch();
  return FT_E_OK;
}
