// The grouped products of a mixture of experts on the 5th-generation tensor cores: C[row, :] = A[row, :] W_e^T for the
// rows of every tile of sorted rows, W_e the tile's expert.
//
// The weights are the 256 rows of a product (M) and the tokens its columns (N, as many as the tile has, rounded up to 32):
// an expert with 260 rows costs 288 columns, not three tiles of 128 rows, and one with eight reads its weights past 32
// columns.  A cluster of two blocks works on a tile (tcgen05 cta_group::2, as gemm_tc_pair.cu: each block holds 128 of the
// weight rows and half of the tokens), one cluster per pair of SMs walks over (token tile, 256 weight rows), weight rows
// fastest, so that the clusters running at one time share a few tokens in L2 and read every weight once.  The ring of
// stages (64 k) and the two accumulators of 256 columns run on from tile to tile.  Weights and tokens have a producer warp
// each: one thread for both set the pace (one instruction more in its loop, a copy to L2 ahead of the ring, made 64 tokens
// 506 us in place of 430).
//
// What counts is bytes in flight: with four stages of 48 KB every size was a third slower than with six of 32, at any number
// of tokens.  So CAP, the tokens of a tile at most, is 64 (11 stages of 20 KB: steps of few tokens are a stream of weights)
// or 320 (six of 36 KB): where experts get some 256 tokens, which a prompt's step of 2,048 with 4 of 32 experts means, a
// tile of 256 would leave half of them with a second one that reads all weights again.  More than 256 tokens are two parts of
// about the same size, an accumulator each (256 and a few: the few cost what some hundred do).
//   * the weight operand is ONE tensor map over all experts' matrices, and the expert moves the box: down the rows (the
//     first matrices, stacked [E F, D]) or along the columns (the second ones, side by side [D, E F]; what a box reads
//     beyond the expert's F columns meets zeros of A, whose map ends at F);
//   * a lane of the accumulator is a weight row, i.e. a column of C, and its columns are tokens: a warp stores 32
//     neighbouring columns of one token at a time.  The first product's epilogue is relu(c)^2 * weight(row) or a gated
//     activation (gate and up are neighbouring lanes, which exchange one of two tokens each) in bfloat16, the second's float.
// The rows of A must lie in sorted order, so the tokens are gathered first (moe_gather_rows).
// Every wait on an mbarrier is bounded as in gemm_tcgen05.cu.
// Bound by the stream of weights up to some 130 rows an expert (32 of 4096 x 3072, 4 chosen, 128 tokens: 2.4 GB in 414 us, 5.9
// TB/s), by that and the products together at 2,048 tokens (0.62 TFLOP in 750 us).  The whole part, 8 / 2,048 tokens: tiles of
// 128 x 256 on one SM and 16 rows on mma.sync 413 / 1,161 us; this with four epilogue warps 284 / 956, with eight 280 / 866.
#include "cluster_common.cuh"
#include <cuda.h>
#include <type_traits>

#include "tc_pair_common.cuh"
#include "tma_host.h"

using namespace ccb;

namespace {

constexpr int kFeatures = 256;     // weight rows of a tile; each block loads 128 of them
constexpr int kTokens = 256;       // tokens of an accumulator at most; each block loads half of them
constexpr int kTokenStep = 32;     // what their number is rounded up to
constexpr int kK = 64;
constexpr int kWBytes = (kFeatures / 2) * kK * 2;   // 16 KB
template <int CAP> struct Ring {
  static constexpr int kParts = (CAP + kTokens - 1) / kTokens;
  static constexpr int kPartBytes = CAP / 4 * kK * 2;         // of the first of two parts, at most
  static constexpr int kBytes = kWBytes + CAP / 2 * kK * 2;   // a stage: the weights, then the tokens
  static constexpr int kStages = CAP == 64 ? 11 : 6;
};
constexpr int kBoxes = 4;          // token copies come in boxes of 16, 32, 64 and 128 rows: at most three make up a block's half
constexpr int kThreads = 352;     // warps: 0 weights, 1 products, 2 .. 9 epilogue, 10 tokens
constexpr int kAcc = 2;            // accumulators of 256 columns in tensor memory

struct TokenMaps {
  CUtensorMap box[kBoxes];   // 16 << i rows
};

struct GroupedTiles {
  const int *e, *r0, *n;   // expert, first sorted row and rows of a token tile; those with rows come first
  int max_tiles, tiles_f;
};

// MODE 0: weight rows at e * F + the tile's, C bfloat16 = relu(c)^2 * row_w;  MODE 1: weight columns at e * F + k, C float;
// MODE 2: as MODE 0 with gate and up rows in turn (F rows an expert, N = F), C bfloat16 [*, N / 2] = glu(gate, up) * row_w
// (ccb::glu_act), or with w_in glu(gate * row_w, up * row_w).
template <int MODE, int CAP>
__global__ void __launch_bounds__(kThreads, 1)
moe_grouped_tc_kernel(const __grid_constant__ TokenMaps tmX, const __grid_constant__ CUtensorMap tmW,
                      void* __restrict__ Cout, int ldc, const float* __restrict__ row_w, const GroupedTiles tiles, int N, int K,
                      int F, const CcbGluAct act, int w_in, int* status) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
  constexpr int kStages = Ring<CAP>::kStages, kBytes = Ring<CAP>::kBytes, XT = Ring<CAP>::kParts,
                kPartBytes = Ring<CAP>::kPartBytes;
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + kStages * kBytes);
  const uint32_t full0 = s32(bars), empty0 = s32(bars + kStages), tfull0 = s32(bars + 2 * kStages),
                 tempty0 = s32(bars + 2 * kStages + 2);
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 2 * kStages + 4);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t rank = cluster_rank();
  const bool leader = rank == 0;
  const int pair = blockIdx.x >> 1, n_pairs = gridDim.x >> 1;
  const int nkb = (K + kK - 1) / kK;
  const int items = tiles.max_tiles * tiles.tiles_f;

  if (threadIdx.x == 0) {
    for (int s = 0; s < kStages; ++s) {
      mbar_init(full0 + 8 * s, 1);
      mbar_init(empty0 + 8 * s, 1);
    }
    for (int b = 0; b < kAcc; ++b) {
      mbar_init(tfull0 + 8 * b, 1);
      mbar_init(tempty0 + 8 * b, 16);   // eight epilogue warps of each block
    }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 1) {   // a warp of EACH block of the pair allocates: the columns are taken in both
    asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(s32(tmem_slot)),
                 "r"((uint32_t)(kAcc * kTokens))
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
  }
  tc_fence_before();
  __syncthreads();
  cluster_sync_all();   // both blocks' barriers exist before anybody signals across
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  pdl_wait();
  if (threadIdx.x == 0) pdl_trigger();

  // every role walks over the same items: (token tile, 256 weight rows); the first token tile without rows ends the walk
  auto columns = [](int n) { return (n + kTokenStep - 1) / kTokenStep * kTokenStep; };
  auto part_columns = [&](int n, int parts, int a) {   // of part a of a tile of n tokens: two parts are as alike as steps allow
    const int all = columns(n), first = parts == 1 ? all : columns((all + 1) / 2);
    return a == 0 ? first : all - first;
  };
  // (the ring's waits have the block's scope: what they order are copies and products, which the barriers count themselves)
  if (warp == 0) {
    if (lane == 0) {  // ---- TMA producer: this block's half of the weight rows ----
      int s = 0, ph = 0;
      bool alive = true;
      const uint32_t full_leader = map_to_rank(full0, 0);
      for (int t = pair; t < items && alive; t += n_pairs) {
        const int ti = t / tiles.tiles_f, tf = t - ti * tiles.tiles_f;
        const int n = min(tiles.n[ti], CAP);
        if (n <= 0) break;
        const int e = tiles.e[ti];
        const int w_row = (MODE != 1 ? e * F : 0) + tf * kFeatures + (int)rank * (kFeatures / 2);
        const int w_col = MODE != 1 ? 0 : e * F;
        const uint32_t bytes = 2 * kWBytes + columns(n) * kK * 2;   // of both blocks, the tokens' copies too
        for (int kb = 0; kb < nkb; ++kb) {
          if (!mbar_wait(empty0 + 8 * s, ph ^ 1)) {
            set_status(status, CCB_ST_WAIT_TIMEOUT);
            alive = false;
            break;
          }
          // the leader expects the bytes of both blocks (see gemm_tc_pair.cu)
          if (leader) mbar_expect_tx(full0 + 8 * s, bytes);
          tma_load_2d_pair(s32(smem + s * kBytes), &tmW, w_col + kb * kK, w_row, full_leader + 8 * s);
          if (++s == kStages) s = 0, ph ^= 1;
        }
      }
    }
  } else if (warp == 10) {
    if (lane == 0) {  // ---- the same for this block's half of the tokens ----
      int s = 0, ph = 0;
      bool alive = true;
      const uint32_t full_leader = map_to_rank(full0, 0);
      for (int t = pair; t < items && alive; t += n_pairs) {
        const int ti = t / tiles.tiles_f;
        const int n = min(tiles.n[ti], CAP);
        if (n <= 0) break;
        const int r0 = tiles.r0[ti];
        // (tiles of one accumulator and of two have loops of their own: conditions inside cost every step of both)
        auto walk = [&](auto parts) {
          constexpr int P = decltype(parts)::value;
          int half[P], x_row[P];
#pragma unroll
          for (int a = 0; a < P; ++a) {
            half[a] = part_columns(n, P, a) / 2;
            x_row[a] = r0 + (a ? part_columns(n, P, 0) : 0) + (int)rank * half[a];
          }
          for (int kb = 0; kb < nkb; ++kb) {
            if (!mbar_wait(empty0 + 8 * s, ph ^ 1)) {
              set_status(status, CCB_ST_WAIT_TIMEOUT);
              alive = false;
              return;
            }
            const uint32_t bar = full_leader + 8 * s, at = s32(smem + s * kBytes) + kWBytes;
#pragma unroll
            for (int a = 0; a < P; ++a) {
              int x = 0;   // (one instruction a box sets the pace: eight boxes of 16 rows halved the rate of full tiles)
#pragma unroll
              for (int b = kBoxes - 1; b >= 0; --b)
                if (half[a] & (16 << b)) {
                  tma_load_2d_pair(at + a * kPartBytes + x * kK * 2, &tmX.box[b], kb * kK, x_row[a] + x, bar);
                  x += 16 << b;
                }
            }
            if (++s == kStages) s = 0, ph ^= 1;
          }
        };
        if (XT == 1 || n <= kTokens) walk(std::integral_constant<int, 1>{});
        else walk(std::integral_constant<int, XT>{});
      }
    }
  } else if (warp == 1) {
    if (lane == 0 && leader) {  // ---- MMA issuer (the leader's): products of M = 256 over both blocks ----
      int s = 0, ph = 0, local = 0;
      bool alive = true;
      for (int t = pair; t < items && alive; t += n_pairs) {
        const int n = min(tiles.n[t / tiles.tiles_f], CAP);
        if (n <= 0) break;
        auto walk = [&](auto parts) {
          constexpr int P = decltype(parts)::value;
          uint32_t idesc[P], acc[P];
#pragma unroll
          for (int a = 0; a < P; ++a) {
            idesc[a] = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(part_columns(n, P, a) >> 3) << 17) |
                       ((uint32_t)(kFeatures >> 4) << 24);
            acc[a] = tmem_base + ((local + a) % kAcc) * kTokens;
            if (!mbar_wait_cluster(tempty0 + 8 * ((local + a) % kAcc), (((local + a) / kAcc) & 1) ^ 1)) return false;
          }
          tc_fence_after();
          for (int kb = 0; kb < nkb; ++kb) {
            if (!mbar_wait(full0 + 8 * s, ph)) return false;
            tc_fence_after();
            const uint64_t da = smem_desc(s32(smem + s * kBytes));
#pragma unroll
            for (int a = 0; a < P; ++a) {
              const uint64_t db = smem_desc(s32(smem + s * kBytes + kWBytes + a * kPartBytes));
#pragma unroll
              for (int k = 0; k < kK / 16; ++k) tc_mma2(acc[a], da + 2 * k, db + 2 * k, idesc[a], (kb > 0 || k > 0) ? 1u : 0u);
            }
            tc_commit2(empty0 + 8 * s);
            if (++s == kStages) s = 0, ph ^= 1;
          }
#pragma unroll
          for (int a = 0; a < P; ++a) tc_commit2(tfull0 + 8 * ((local + a) % kAcc));
          local += P;
          return true;
        };
        alive = XT == 1 || n <= kTokens ? walk(std::integral_constant<int, 1>{}) : walk(std::integral_constant<int, XT>{});
        if (!alive) set_status(status, CCB_ST_WAIT_TIMEOUT);
      }
    }
  } else {  // ---- epilogue: this block's 128 weight rows (lanes), all tokens of the tile (columns) ----
    // two warps a quarter of the lanes, which take 32 tokens in turn (one warp each left a third of a tile's time exposed
    // where both accumulators are taken)
    const int q = warp & 3, turn = (warp - 2) >> 2;
    int local = 0;
    bool alive = true;
    for (int t = pair, n0 = 0; t < items && alive; ++local) {   // an accumulator at a time: tokens n0 .. of item t
      const int ti = t / tiles.tiles_f, tf = t - ti * tiles.tiles_f;
      const int n_tile = min(tiles.n[ti], CAP);
      if (n_tile <= 0) break;
      const int n = min(n_tile - n0, XT == 1 || n_tile <= kTokens ? kTokens : part_columns(n_tile, 2, n0 ? 1 : 0));
      const int buf = local % kAcc;
      alive = mbar_wait_cluster(tfull0 + 8 * buf, (local / kAcc) & 1);
      if (!alive) {
        if (lane == 0) set_status(status, CCB_ST_WAIT_TIMEOUT);
        break;
      }
      tc_fence_after();
      const size_t g0 = (size_t)tiles.r0[ti] + n0;
      const int col = tf * kFeatures + (int)rank * (kFeatures / 2) + q * 32 + lane;   // this lane's column of the product
      const uint32_t taddr = tmem_base + buf * kTokens + ((uint32_t)(q * 32) << 16);
#pragma unroll 1
      for (int c0 = 32 * turn; c0 < n; c0 += 64) {
        uint32_t v[32];
        tc_ld32(taddr + c0, v);
        tc_wait_ld();
        const float my_w = MODE != 1 && c0 + lane < n ? row_w[g0 + c0 + lane] : 1.f;
        if (MODE == 1) {
          float* dst = (float*)Cout + (g0 + c0) * ldc + col;
#pragma unroll
          for (int j = 0; j < 32; ++j)
            if (c0 + j < n && col < N) dst[(size_t)j * ldc] = __uint_as_float(v[j]);
        } else if (MODE == 0) {
          __nv_bfloat16* dst = (__nv_bfloat16*)Cout + (g0 + c0) * ldc + col;
#pragma unroll
          for (int j = 0; j < 32; ++j) {
            const float w = __shfl_sync(0xffffffffu, my_w, j), a = fmaxf(__uint_as_float(v[j]), 0.f);
            if (c0 + j < n && col < N) dst[(size_t)j * ldc] = __float2bfloat16_rn(a * a * w);
          }
        } else {   // columns (2 f, 2 f + 1) are gate f and up f: the even lane takes token j, the odd one token j + 1
          const int odd = lane & 1;
          __nv_bfloat16* dst = (__nv_bfloat16*)Cout + (g0 + c0 + odd) * ldc + (col >> 1);
          const bool mine = (col | 1) < N;
          auto one = [&](int j) {
            const float w = __shfl_sync(0xffffffffu, my_w, j + odd);
            const float wi = w_in ? w : 1.f, wo = w_in ? 1.f : w;
            const float a = __uint_as_float(v[j]), b = __uint_as_float(v[j + 1]);
            const float got = __shfl_xor_sync(0xffffffffu, odd ? a : b, 1);   // what the other lane has of this lane's token
            return glu_act(act, (odd ? got : a) * wi, (odd ? b : got) * wi) * wo;
          };
          if (c0 + 32 <= n) {   // (no condition a token: the activations of several run side by side)
#pragma unroll
            for (int j = 0; j < 32; j += 2) {
              const float y = one(j);
              if (mine) dst[(size_t)j * ldc] = __float2bfloat16_rn(y);
            }
          } else {
#pragma unroll
            for (int j = 0; j < 32; j += 2) {
              const float y = one(j);
              if (mine && c0 + j + odd < n) dst[(size_t)j * ldc] = __float2bfloat16_rn(y);
            }
          }
        }
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) {   // this warp's quarter of this block's accumulator is free again: the leader counts sixteen
        if (leader) mbar_arrive(tempty0 + 8 * buf);
        else mbar_arrive_remote(map_to_rank(tempty0 + 8 * buf, 0));
      }
      n0 += n;
      if (n0 >= n_tile) n0 = 0, t += n_pairs;
    }
  }
  tc_fence_before();
  __syncthreads();
  cluster_sync_all();   // nobody leaves while the other block may still signal it or read its shared memory
  if (warp == 1) {
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"((uint32_t)(kAcc * kTokens))
                 : "memory");
  }
}

// out[pos, :] = x[src_row[pos], :]: the tokens in sorted order, 16 bytes a thread and step
__global__ void __launch_bounds__(256)
moe_gather_rows_kernel(uint4* __restrict__ out, const uint4* __restrict__ x, const int* __restrict__ src_row, int ldx16,
                       int row16, size_t total) {
  ccb::pdl_begin();
  for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += (size_t)gridDim.x * blockDim.x) {
    const size_t pos = i / row16;
    const int c = (int)(i - pos * row16);
    out[i] = x[(size_t)src_row[pos] * ldx16 + c];
  }
}

template <int MODE, int CAP>
int launch(const TokenMaps& tmX, const CUtensorMap& tmW, void* C, int ldc, const float* row_w, const GroupedTiles& tiles, int N,
           int K, int F, const CcbGluAct& act, int w_in, int sms, int* status, cudaStream_t stream) {
  constexpr size_t smem = (size_t)Ring<CAP>::kStages * Ring<CAP>::kBytes + (2 * Ring<CAP>::kStages + 4) * 8 + 16 + 1024;
  static bool configured = false;
  if (!configured) {
    cudaError_t e = cudaFuncSetAttribute(moe_grouped_tc_kernel<MODE, CAP>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return (int)e;
    configured = true;
  }
  const int items = tiles.max_tiles * tiles.tiles_f;
  const int pairs = items < sms / 2 ? items : sms / 2;
  ccb_launch_cluster(false, 2, moe_grouped_tc_kernel<MODE, CAP>, dim3(2 * pairs), dim3(kThreads), smem, stream, tmX, tmW, C, ldc,
                     row_w, tiles, N, K, F, act, w_in, status);
  return ccb_launch_status();
}

}  // namespace

// bfloat16 rows of `width` elements (a multiple of 8), x rows at ldx: out [rows, width] = x[src_row[.]]
CCB_API int ccb_moe_gather_rows(void* out, const void* x, const int* src_row, int rows, int width, int ldx,
                                cudaStream_t stream) {
  if (rows <= 0) return 0;
  if (width <= 0 || (width & 7) || (ldx & 7) || (reinterpret_cast<uintptr_t>(out) & 15) ||
      (reinterpret_cast<uintptr_t>(x) & 15))
    return CCB_REFUSE_SIZE;
  const size_t total = (size_t)rows * (width / 8);
  const int blocks = (int)((total + 255) / 256 < 65535 * 8 ? (total + 255) / 256 : 65535 * 8);
  ccb_launch(moe_gather_rows_kernel, dim3(blocks), dim3(256), 0, stream, (uint4*)out, (const uint4*)x, src_row, ldx / 8,
             width / 8, total);
  return ccb_launch_status();
}

// The tiles are those of moe_sort with BM = tile_rows, 64 or 320.  A [rows, K] holds the sorted rows (contiguous rows of lda).
// mode 0: W = the first matrices stacked [w_rows, K] (expert e at row e * F), C bfloat16 [rows, N = F] with
// relu(.)^2 * row_w;  mode 1: W = the second matrices side by side [N, w_cols] (expert e at column e * F, K = F),
// C float [rows, N];  mode 2: W = the first matrices stacked with every expert's gate and up rows in turn (F rows an
// expert, N = F), C bfloat16 [rows, N / 2] = glu(gate, up) * row_w, or with w_in glu(gate * row_w, up * row_w); limit,
// alpha, shift, cubic: which glu (CcbGluAct).  sms: how many SMs the device has.
CCB_API int ccb_moe_grouped_tc(const void* A, int lda, int rows, const void* W, int ldw, int w_rows, int w_cols,
                               void* C, int ldc, const float* row_w, const int* tile_e, const int* tile_r0,
                               const int* tile_n, int max_tiles, int N, int K, int F, int mode, float limit, float alpha,
                               float shift, float cubic, int w_in, int tile_rows, int sms, int* status,
                               cudaStream_t stream) {
  if (tile_rows != 64 && tile_rows != 320) return CCB_REFUSE_SIZE;
  if (max_tiles <= 0 || N <= 0 || rows <= 0) return 0;
  if (K <= 0 || (K & 7) || (F & 7) || (lda & 7) || (ldw & 7) || mode < 0 || mode > 2 || (mode == 2 && (N & 1)) || sms < 2 ||
      (long long)max_tiles * ((N + kFeatures - 1) / kFeatures) > 0x7fffffffll ||
      (reinterpret_cast<uintptr_t>(A) & 15) || (reinterpret_cast<uintptr_t>(W) & 15))
    return CCB_REFUSE_SIZE;
  const CcbGluAct ga{limit, alpha, shift, cubic};
  const GroupedTiles tiles{tile_e, tile_r0, tile_n, max_tiles, (N + kFeatures - 1) / kFeatures};
  TokenMaps tmX;
  CUtensorMap tmW;
  for (int i = 0; i < kBoxes; ++i)
    if (!ccb_tensor_map_2d(A, rows, K, lda, kK, 16 << i, &tmX.box[i])) return CCB_REFUSE_ARG;
  if (!ccb_tensor_map_2d(W, w_rows, w_cols, ldw, kK, kFeatures / 2, &tmW)) return CCB_REFUSE_ARG;
#define CCB_GROUPED(MODE)                                                                                             \
  (tile_rows == 64 ? launch<MODE, 64>(tmX, tmW, C, ldc, row_w, tiles, N, K, F, ga, w_in, sms, status, stream)        \
                   : launch<MODE, 320>(tmX, tmW, C, ldc, row_w, tiles, N, K, F, ga, w_in, sms, status, stream))
  if (mode == 2) return CCB_GROUPED(2);
  if (mode == 0) return CCB_GROUPED(0);
  return CCB_GROUPED(1);
#undef CCB_GROUPED
}
