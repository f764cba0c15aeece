// The grouped products of a mixture of experts on the 5th-generation tensor cores: C[row, :] = A[row, :] W_e^T for the
// rows of every tile of sorted rows, W_e the tile's expert.
//
// The weights are the 256 rows of a product (M) and the tokens its columns (N, as many as the tile has, rounded up to 32):
// an expert with 260 rows costs 288 columns, not three tiles of 128 rows, and one with eight reads its weights past 32
// columns.  A cluster of two blocks works on a tile (tcgen05 cta_group::2, as gemm_tc_pair.cu: each block holds 128 of the
// weight rows and half of the tokens), one cluster per pair of SMs walks over (token tile, 256 weight rows), weight rows
// fastest, so that the clusters running at one time share a few tokens in L2 and read every weight once.  The ring of
// stages (64 k) runs on from tile to tile, and so does tensor memory: its 512 columns are a ring of sixteen slots of 32, a tile
// takes as many as it has columns, and the next one's products begin as soon as the slots that it needs have been read
// (`slot_ring.h`).  (Two
// accumulators of 256 columns, both of which a tile of more tokens took, left its whole epilogue without products beside it.)
// Weights and tokens have a producer warp
// each: one thread for both set the pace (one instruction more in its loop, a copy to L2 ahead of the ring, made 64 tokens
// 506 us in place of 430).
//
// What counts is bytes in flight: with four stages of 48 KB every size was a third slower than with six of 32, at any number
// of tokens.  So CAP, the tokens of a tile at most, is 64 (11 stages of 20 KB: steps of few tokens are a stream of weights)
// or 320 (six of 36 KB): where experts get some 256 tokens, which a prompt's step of 2,048 with 4 of 32 experts means, a
// tile of 256 would leave half of them with a second one that reads all weights again.  A product has neighbouring columns and 256
// at most, so a tile is up to three of them (`TileParts`); each block of the pair holds one half of the tile's tokens, and the
// columns of a product are some tokens of the one half and then as many of the other.
//   * the weight operand is ONE tensor map over all experts' matrices, and the expert moves the box: down the rows (the
//     first matrices, stacked [E F, D]) or along the columns (the second ones, side by side [D, E F]; what a box reads
//     beyond the expert's F columns meets zeros of A, whose map ends at F);
//   * a lane of the accumulator is a weight row, i.e. a column of C, and its columns are tokens: a warp stores 32
//     neighbouring columns of one token at a time.  The first product's epilogue is relu(c)^2 * weight(row) or a gated
//     activation (gate and up are neighbouring lanes, which exchange one of two tokens each) in bfloat16, the second's float.
// The rows of A must lie in sorted order, so the tokens are gathered first (moe_gather_rows).
// Every wait on an mbarrier is bounded as in gemm_tcgen05.cu.
// Bound by the stream of weights up to some 130 rows an expert (32 of 4096 x 3072, 4 chosen, 128 tokens: 2.4 GB in 414 us, 5.9
// TB/s), by that and the products together at 2,048 tokens (0.62 TFLOP in 580 us).  The whole part, 8 / 2,048 tokens: tiles of
// 128 x 256 on one SM and 16 rows on mma.sync 413 / 1,161 us; this with two accumulators and eight epilogue warps 281 / 898, with the
// ring of slots 279 / 779 (width 2,048: 125 / 377 and 121 / 318; 128 to 1,100 tokens the same within 2 per cent).  A warp's signal that
// a slot has been read does not wait for its stores: what it orders is a read of tensor memory, which tcgen05.wait::ld and the fence
// have ended (with a releasing one, 1,100 tokens of width 2,048 took 127 us in the first product, 109 so).
#include "cluster_common.cuh"
#include <cuda.h>
#include <type_traits>

#include "slot_ring.h"
#include "tc_pair_common.cuh"
#include "tma_host.h"

using namespace ccb;

namespace {

constexpr int kFeatures = 256;     // weight rows of a tile; each block loads 128 of them
constexpr int kTokenStep = 32;     // what the number of a tile's tokens is rounded up to; each block loads half of them
constexpr int kK = 64;
constexpr int kWBytes = (kFeatures / 2) * kK * 2;   // 16 KB
template <int CAP> struct Ring {
  static constexpr int kBytes = kWBytes + CAP / 2 * kK * 2;   // a stage: the weights, then the tokens
  static constexpr int kStages = CAP == 64 ? 11 : 6;
};
constexpr int kBoxes = 4;          // token copies come in boxes of 16, 32, 64 and 128 rows: at most three make up a block's half
constexpr int kThreads = 352;     // warps: 0 weights, 1 products, 2 .. 9 epilogue, 10 tokens

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
  constexpr int kStages = Ring<CAP>::kStages, kBytes = Ring<CAP>::kBytes;
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + kStages * kBytes);
  const uint32_t full0 = s32(bars), empty0 = s32(bars + kStages), tfull0 = s32(bars + 2 * kStages),
                 tempty0 = s32(bars + 2 * kStages + kSlots);   // of a tile (in turn), of a slot
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 2 * kStages + 2 * kSlots);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t rank = cluster_rank();
  const bool leader = rank == 0;
  const int pair = blockIdx.x >> 1, n_pairs = gridDim.x >> 1;
  const int nkb = (K + kK - 1) / kK;
  const int items = tiles.max_tiles * tiles.tiles_f;

  if (warp == 0) {   // a lane a barrier of each kind
    if (lane < kStages) {
      mbar_init(full0 + 8 * lane, 1);
      mbar_init(empty0 + 8 * lane, 1);
    }
    if (lane < kSlots) {
      mbar_init(tfull0 + 8 * lane, 1);
      mbar_init(tempty0 + 8 * lane, 16);   // eight epilogue warps of each block
    }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 1) {   // a warp of EACH block of the pair allocates: the columns are taken in both
    asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(s32(tmem_slot)),
                 "r"((uint32_t)(kSlots * kTokenStep))
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

  // every role walks over the same items: (token tile, 256 weight rows); the first token tile without rows ends the walk.  Of
  // wide tiles an item is asked for one ahead, since nobody should stop between two of them (2,048 tokens: 406 -> 399 us in the
  // first product); a stream of weights alone has no use for it (8 tokens 169.6 with, 169.0 without).
  constexpr bool kAhead = CAP != 64;
  struct Item {
    int tf, e, r0, n;
  };
  auto item = [&](int t) {
    Item x{0, 0, 0, 0};
    if (t < items) {
      const int ti = t / tiles.tiles_f;
      x = Item{t - ti * tiles.tiles_f, tiles.e[ti], tiles.r0[ti], min(tiles.n[ti], CAP)};
    }
    return x;
  };
  auto columns = [](int n) { return (n + kTokenStep - 1) / kTokenStep * kTokenStep; };
  // (the ring's waits have the block's scope: what they order are copies and products, which the barriers count themselves)
  if (warp == 0) {
    if (lane == 0) {  // ---- TMA producer: this block's half of the weight rows ----
      int s = 0, ph = 0;
      bool alive = true;
      const uint32_t full_leader = map_to_rank(full0, 0);
      Item now = item(pair), next = now;
      for (int t = pair; now.n > 0 && alive; t += n_pairs, now = kAhead ? next : item(t)) {
        if (kAhead) next = item(t + n_pairs);
        const int w_row = (MODE != 1 ? now.e * F : 0) + now.tf * kFeatures + (int)rank * (kFeatures / 2);
        const int w_col = MODE != 1 ? 0 : now.e * F;
        const uint32_t bytes = 2 * kWBytes + columns(now.n) * kK * 2;   // of both blocks, the tokens' copies too
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
      Item now = item(pair), next = now;
      for (int t = pair; now.n > 0 && alive; t += n_pairs, now = kAhead ? next : item(t)) {
        if (kAhead) next = item(t + n_pairs);
        const int half = columns(now.n) / 2, x_row = now.r0 + (int)rank * half;
        for (int kb = 0; kb < nkb; ++kb) {
          if (!mbar_wait(empty0 + 8 * s, ph ^ 1)) {
            set_status(status, CCB_ST_WAIT_TIMEOUT);
            alive = false;
            break;
          }
          const uint32_t bar = full_leader + 8 * s, at = s32(smem + s * kBytes) + kWBytes;
          int x = 0;   // (one instruction a box sets the pace: eight boxes of 16 rows halved the rate of full tiles)
#pragma unroll
          for (int b = kBoxes - 1; b >= 0; --b)
            if (half & (16 << b)) {
              tma_load_2d_pair(at + x * kK * 2, &tmX.box[b], kb * kK, x_row + x, bar);
              x += 16 << b;
            }
          if (++s == kStages) s = 0, ph ^= 1;
        }
      }
    }
  } else if (warp == 1) {
    if (lane == 0 && leader) {  // ---- MMA issuer (the leader's): products of M = 256 over both blocks ----
      int s = 0, ph = 0, local = 0;
      SlotRing ring;
      uint32_t used = 0;   // a bit a slot: how often it has been used, its last place
      bool alive = true;
      Item now = item(pair), next = now;
      for (int t = pair; now.n > 0 && alive; t += n_pairs, now = kAhead ? next : item(t), ++local) {
        if (kAhead) next = item(t + n_pairs);
        const int slots = columns(now.n) / kTokenStep;
        ring.enter(slots);
        const int at = ring.at;
        for (int i = ring.first_waited(slots); i < ring.end_waited(slots) && alive; ++i) {
          const int b = (at + i) % kSlots;
          alive = mbar_wait_cluster(tempty0 + 8 * b, (used >> b & 1) ^ 1);
        }
        used ^= slot_bits(at, slots);
        if (!alive) {
          set_status(status, CCB_ST_WAIT_TIMEOUT);
          break;
        }
        tc_fence_after();
        const TileParts parts(at, slots);
        auto walk = [&](auto count) {
          constexpr int P = decltype(count)::value;
          uint32_t idesc[P], acc[P], from[P];
#pragma unroll
          for (int a = 0, first = 0; a < P; first += parts.len[a++]) {
            idesc[a] = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(parts.len[a] * kTokenStep >> 3) << 17) |
                       ((uint32_t)(kFeatures >> 4) << 24);
            acc[a] = tmem_base + (at + first) % kSlots * kTokenStep;
            from[a] = first * (kTokenStep / 2) * kK * 2;
          }
          for (int kb = 0; kb < nkb; ++kb) {
            if (!mbar_wait(full0 + 8 * s, ph)) return false;
            tc_fence_after();
            const uint64_t da = smem_desc(s32(smem + s * kBytes));
#pragma unroll
            for (int a = 0; a < P; ++a) {
              const uint64_t db = smem_desc(s32(smem + s * kBytes + kWBytes) + from[a]);
#pragma unroll
              for (int k = 0; k < kK / 16; ++k) tc_mma2(acc[a], da + 2 * k, db + 2 * k, idesc[a], (kb > 0 || k > 0) ? 1u : 0u);
            }
            tc_commit2(empty0 + 8 * s);
            if (++s == kStages) s = 0, ph ^= 1;
          }
          tc_commit2(tfull0 + 8 * (local % kSlots));
          return true;
        };
        const int count = CAP <= kMostSlots * kTokenStep ? 1 : parts.count();
        alive = count == 1   ? walk(std::integral_constant<int, 1>{})
                : count == 2 ? walk(std::integral_constant<int, 2>{})
                             : walk(std::integral_constant<int, 3>{});
        if (!alive) set_status(status, CCB_ST_WAIT_TIMEOUT);
        ring.leave(slots);
      }
    }
  } else {  // ---- epilogue: this block's 128 weight rows (lanes), all tokens of the tile (columns) ----
    // two warps a quarter of the lanes, which take a slot in turn
    const int q = warp & 3, turn = (warp - 2) >> 2;
    int local = 0;
    SlotRing ring;
    Item now = item(pair), next = now;
    for (int t = pair; now.n > 0; t += n_pairs, now = kAhead ? next : item(t), ++local) {
      if (kAhead) next = item(t + n_pairs);
      const int n = now.n;
      if (!mbar_wait_cluster(tfull0 + 8 * (local % kSlots), (local / kSlots) & 1)) {
        if (lane == 0) set_status(status, CCB_ST_WAIT_TIMEOUT);
        break;
      }
      tc_fence_after();
      const int slots = columns(n) / kTokenStep, half = slots * (kTokenStep / 2);
      ring.enter(slots);
      const int at = ring.at;
      const TileParts parts(at, slots);
      const size_t g0 = (size_t)now.r0;
      const int col = now.tf * kFeatures + (int)rank * (kFeatures / 2) + q * 32 + lane;   // this lane's column of the product
      auto done_with = [&](int i) {   // the leader counts all sixteen warps, so that none is a turn of the ring behind
        const uint32_t bar = tempty0 + 8 * ((at + i) % kSlots);
        if (leader) mbar_arrive(bar);
        else mbar_arrive_remote_relaxed(map_to_rank(bar, 0));
      };
      if (lane == 0)
        for (int i = turn ^ 1; i < slots; i += 2) done_with(i);
#pragma unroll 1
      for (int i = turn; i < slots; i += 2) {
        const int b = (at + i) % kSlots;
        // the tokens of the slot's columns, sixteen neighbours twice: of the product's columns the first half are tokens of the
        // tile's first half
        int tok[2];
        {
          const int second = parts.len[0], third = second + parts.len[1];   // where the products begin
          const int first = i < second ? 0 : i < third ? second : third;
          const int width = (i < second ? parts.len[0] : i < third ? parts.len[1] : parts.len[2]) * (kTokenStep / 2);   // of a half
#pragma unroll
          for (int x = 0; x < 2; ++x) {
            const int j = (i - first) * kTokenStep + 16 * x;
            tok[x] = first * (kTokenStep / 2) + (j < width ? j : half + j - width);
          }
        }
        const int mine = tok[lane >> 4] + (lane & 15);
        const float my_w = MODE != 1 && mine < n ? row_w[g0 + mine] : 1.f;
        uint32_t v[32];
        tc_ld32(tmem_base + b * kTokenStep + ((uint32_t)(q * 32) << 16), v);
        tc_wait_ld();
        tc_fence_before();
        __syncwarp();
        if (lane == 0) done_with(i);
        if (MODE == 2 && tok[0] + 16 <= n && tok[1] + 16 <= n) {   // (no condition a token: the activations of many run side by side)
          const int odd = lane & 1;
          __nv_bfloat16* dst[2];
#pragma unroll
          for (int x = 0; x < 2; ++x) dst[x] = (__nv_bfloat16*)Cout + (g0 + tok[x] + odd) * ldc + (col >> 1);
          const bool mine_col = (col | 1) < N;
#pragma unroll
          for (int j = 0; j < 32; j += 2) {
            const float w = __shfl_sync(0xffffffffu, my_w, j + odd);
            const float wi = w_in ? w : 1.f, wo = w_in ? 1.f : w;
            const float a = __uint_as_float(v[j]), c = __uint_as_float(v[j + 1]);
            const float got = __shfl_xor_sync(0xffffffffu, odd ? a : c, 1);
            const float y = glu_act(act, (odd ? got : a) * wi, (odd ? c : got) * wi) * wo;
            if (mine_col) dst[j >> 4][(size_t)(j & 15) * ldc] = __float2bfloat16_rn(y);
          }
          continue;
        }
#pragma unroll
        for (int x = 0; x < 2; ++x) {
          const size_t row = g0 + tok[x];
          const int left = n - tok[x];   // of the sixteen tokens
          if (left <= 0) continue;   // (columns without tokens, of which a step of few has most)
          if (MODE == 1) {
            float* dst = (float*)Cout + row * ldc + col;
#pragma unroll
            for (int j = 0; j < 16; ++j) {
              if (j >= left) break;
              if (col < N) dst[(size_t)j * ldc] = __uint_as_float(v[16 * x + j]);
            }
          } else if (MODE == 0) {
            __nv_bfloat16* dst = (__nv_bfloat16*)Cout + row * ldc + col;
#pragma unroll
            for (int j = 0; j < 16; ++j) {
              if (j >= left) break;
              const float w = __shfl_sync(0xffffffffu, my_w, 16 * x + j), a = fmaxf(__uint_as_float(v[16 * x + j]), 0.f);
              if (col < N) dst[(size_t)j * ldc] = __float2bfloat16_rn(a * a * w);
            }
          } else {   // columns (2 f, 2 f + 1) are gate f and up f: the even lane takes token j, the odd one token j + 1
            const int odd = lane & 1;
            __nv_bfloat16* dst = (__nv_bfloat16*)Cout + (row + odd) * ldc + (col >> 1);
            const bool mine_col = (col | 1) < N;
            auto one = [&](int j) {
              const float w = __shfl_sync(0xffffffffu, my_w, 16 * x + j + odd);
              const float wi = w_in ? w : 1.f, wo = w_in ? 1.f : w;
              const float a = __uint_as_float(v[16 * x + j]), c = __uint_as_float(v[16 * x + j + 1]);
              const float got = __shfl_xor_sync(0xffffffffu, odd ? a : c, 1);   // what the other lane has of this lane's token
              return glu_act(act, (odd ? got : a) * wi, (odd ? c : got) * wi) * wo;
            };
#pragma unroll
            for (int j = 0; j < 16; j += 2) {
              if (j >= left) break;
              const float y = one(j);
              if (mine_col && j + odd < left) dst[(size_t)j * ldc] = __float2bfloat16_rn(y);
            }
          }
        }
      }
      ring.leave(slots);
    }
  }
  tc_fence_before();
  __syncthreads();
  cluster_sync_all();   // nobody leaves while the other block may still signal it or read its shared memory
  if (warp == 1) {
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"((uint32_t)(kSlots * kTokenStep))
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
  constexpr size_t smem = (size_t)Ring<CAP>::kStages * Ring<CAP>::kBytes + (2 * Ring<CAP>::kStages + 2 * kSlots) * 8 + 16 + 1024;
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
