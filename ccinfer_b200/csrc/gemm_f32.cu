// True 32-bit matrix product for the float path: C[M, N] = A[M, K] * W[N, K]^T.
//
// IEEE float fused multiply-adds on the CUDA cores: no tensor cores, no TF32,
// no reduced-precision mode of any library (7QiC/ccInfer runs this product in
// cuBLAS with float accumulation, src/backend/cuda/cuda_backend.cpp:82-108).
// The k range is cut into eight segments of equal length (`segment_of`, from K
// alone).  A segment of an output element is one accumulation chain over its k
// in ascending order, and the eight sums are added in ascending order, whatever
// kernel or tile shape runs, so a row's result does not depend on how many other
// rows are in the batch.  Any M, N, K.
//
// Two kernels:
//   rows   M <= 16: the product is a stream of W.  A block takes 16 rows of W and its eight half-warps a segment
//          each, so that 64 blocks already keep eight streams an SM going: cp.async into a ring that each warp owns,
//          a lane per row of W, A's values broadcast from the same ring.
//   tiles  M > 16: BM x 128 tiles, 8 x 8 places a thread whatever BM is (six 16-byte reads of shared memory for 64
//          multiply-adds; with 4 x 8 places the reads set the pace), two multiply-adds an instruction (fma.rn.f32x2).
//          Where the tiles do not fill the machine a cluster of eight blocks takes a tile, a segment each, and adds up
//          through distributed shared memory.
// What bounds them: the rows kernel the stream of W (2 x 16,384 x 2,048: 34 us, 3.9 TB/s; 2 x 32,000 x 2,048: 57 us, 4.6
// TB/s) until many rows make it the reads of A (16 x 16,384 x 2,048: 66 us); the tiles kernel the multiply-adds (300 x
// 16,384 x 2,048: 515 us, 39 TFLOP/s; 1,024 rows: 48 TFLOP/s of 72).  One tile kernel for every M, without segments or
// pipelining, took 562 us on average for the products of 2-3 rows of a model of width 2,048 and 771 us for those of some
// 200 rows; a call of that model (two prompts of some 100 tokens, three more tokens each) went from 22.7 to 3.0 ms.
#include "cluster_common.cuh"
#include "mma_common.cuh"

using namespace ccb;

namespace {

constexpr int kSegments = 8;

// length of a segment: a multiple of 32
__host__ __device__ __forceinline__ int segment_of(int K) { return ((K + 32 * kSegments - 1) / (32 * kSegments)) * 32; }

// 16 bytes global -> shared of which the first `bytes` are read and the others become zeros
__device__ __forceinline__ void copy16(uint32_t dst, const float* src, int bytes) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(dst), "l"(src), "r"(bytes));
}
__device__ __forceinline__ void copy4(uint32_t dst, const float* src, int bytes) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;\n" ::"r"(dst), "l"(src), "r"(bytes));
}

// ---------------------------------------------------------------------------------------------
constexpr int kRowWarps = 4;     // two segments each
constexpr int kRowW = 16;        // rows of W a block
constexpr int kRowK = 32;        // k of a stage
constexpr int kRowPitch = 36;    // floats: a lane per row reads 16 bytes without bank conflicts

template <int MR> struct RowsStage {
  static constexpr int kA = MR * kRowK + 4;                       // floats of A of one segment (4: other banks for the other one)
  static constexpr int kFloats = 2 * kRowW * kRowPitch + 2 * kA;
  static constexpr int kStages = MR > 8 ? 3 : 4;
  static constexpr int kBytes = kRowWarps * kStages * kFloats * 4;   // (two blocks an SM)
};

template <int MR>
__global__ void __launch_bounds__(kRowWarps * 32)
gemm_f32_rows_kernel(float* __restrict__ C, const float* __restrict__ A, const float* __restrict__ W, int M, int N, int K,
                     int lda, int ldw, int ldc, long long sa, long long sw, long long sc, int vec) {
  ccb::pdl_begin();
  using St = RowsStage<MR>;
  constexpr int S = St::kStages;
  extern __shared__ __align__(16) float smem[];
  C += (size_t)blockIdx.z * sc;
  A += (size_t)blockIdx.z * sa;
  W += (size_t)blockIdx.z * sw;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int n0 = blockIdx.x * kRowW;
  const int seg = segment_of(K), k_seg = 2 * warp * seg;   // of the warp's first segment
  const int tiles = seg / kRowK;
  float* ring = smem + warp * S * St::kFloats;

  auto fetch = [&](int tile, int st) {
    float* w_s = ring + st * St::kFloats;
    float* a_s = w_s + 2 * kRowW * kRowPitch;
    if (tile < tiles) {
      if (vec) {
#pragma unroll
        for (int i = 0; i < 8; ++i) {          // 2 segments x 16 rows x 8 pieces
          const int idx = lane + 32 * i, half = idx >> 7, row = (idx >> 3) & 15, c = idx & 7;
          const int k = k_seg + half * seg + tile * kRowK + c * 4;
          const int bytes = n0 + row < N ? max(0, min(16, 4 * (K - k))) : 0;
          copy16(smem_u32(w_s + (half * kRowW + row) * kRowPitch + c * 4), bytes ? W + (size_t)(n0 + row) * ldw + k : W, bytes);
        }
#pragma unroll
        for (int i = 0; i < (MR * 16 + 31) / 32; ++i) {
          const int idx = lane + 32 * i, half = idx / (MR * 8), m = (idx >> 3) % MR, c = idx & 7;
          const int k = k_seg + half * seg + tile * kRowK + c * 4;
          const int bytes = m < M ? max(0, min(16, 4 * (K - k))) : 0;
          copy16(smem_u32(a_s + half * St::kA + m * kRowK + c * 4), bytes ? A + (size_t)m * lda + k : A, bytes);
        }
      } else {
        for (int idx = lane; idx < 2 * kRowW * kRowK; idx += 32) {
          const int half = idx >> 9, row = (idx >> 5) & 15, c = idx & 31;
          const int k = k_seg + half * seg + tile * kRowK + c;
          const int bytes = n0 + row < N && k < K ? 4 : 0;
          copy4(smem_u32(w_s + (half * kRowW + row) * kRowPitch + c), bytes ? W + (size_t)(n0 + row) * ldw + k : W, bytes);
        }
        for (int idx = lane; idx < 2 * MR * kRowK; idx += 32) {
          const int half = idx / (MR * kRowK), m = (idx >> 5) % MR, c = idx & 31;
          const int k = k_seg + half * seg + tile * kRowK + c;
          const int bytes = m < M && k < K ? 4 : 0;
          copy4(smem_u32(a_s + half * St::kA + m * kRowK + c), bytes ? A + (size_t)m * lda + k : A, bytes);
        }
      }
    }
    cp_async_commit();   // (an empty group keeps the count)
  };

  float acc[MR];
#pragma unroll
  for (int m = 0; m < MR; ++m) acc[m] = 0.f;
#pragma unroll
  for (int s = 0; s < S - 1; ++s) fetch(s, s);
  const int row = lane & 15, half = lane >> 4;
  int st = 0;
  for (int tile = 0; tile < tiles; ++tile) {
    cp_async_wait<S - 2>();
    __syncwarp();   // the stage is there for every lane, and every lane has left the one that is written next
    fetch(tile + S - 1, st == 0 ? S - 1 : st - 1);
    const float* w_s = ring + st * St::kFloats + (half * kRowW + row) * kRowPitch;
    const float* a_s = ring + st * St::kFloats + 2 * kRowW * kRowPitch + half * St::kA;
#pragma unroll
    for (int c = 0; c < kRowK / 4; ++c) {
      const float4 w = *reinterpret_cast<const float4*>(w_s + 4 * c);
#pragma unroll
      for (int m = 0; m < MR; ++m) {
        const float4 a = *reinterpret_cast<const float4*>(a_s + m * kRowK + 4 * c);
        acc[m] = fmaf(a.x, w.x, acc[m]);
        acc[m] = fmaf(a.y, w.y, acc[m]);
        acc[m] = fmaf(a.z, w.z, acc[m]);
        acc[m] = fmaf(a.w, w.w, acc[m]);
      }
    }
    st = st + 1 == S ? 0 : st + 1;
  }
  cp_async_wait<0>();
  __syncthreads();   // every ring has been read: its memory takes the segments' sums
  float* sums = smem;   // [segment][MR][16]
#pragma unroll
  for (int m = 0; m < MR; ++m) sums[((2 * warp + half) * MR + m) * kRowW + row] = acc[m];
  __syncthreads();
  for (int i = threadIdx.x; i < MR * kRowW; i += kRowWarps * 32) {
    const int m = i / kRowW, n = n0 + i % kRowW;
    if (m >= M || n >= N) continue;
    float total = sums[i];
#pragma unroll
    for (int s = 1; s < kSegments; ++s) total += sums[s * MR * kRowW + i];
    C[(size_t)m * ldc + n] = total;
  }
}

// ---------------------------------------------------------------------------------------------
constexpr int kTileK = 16;
constexpr int kTileN = 128;
constexpr int TM = 8;            // rows a thread
constexpr int kWPitch = kTileN + 4;

template <int BM> struct TileShape {
  static constexpr int kThreads = 2 * BM;
  static constexpr int kBlocks = BM == 128 ? 1 : BM == 64 ? 3 : 6;   // an SM, so that no register spills
  static constexpr int kPitch = BM + 4;
  static constexpr int kA = kTileK * kPitch;                       // floats of a stage
  static constexpr int kW = kTileK * kWPitch;
  static constexpr int kTotals = BM * kTileN;                      // a segment's tile, or the total so far
  static constexpr int kBytes = (2 * (kA + kW) + kTotals) * 4;
};

__device__ __forceinline__ unsigned long long twice(float x) {
  unsigned long long r;
  asm("mov.b64 %0, {%1, %1};" : "=l"(r) : "f"(x));
  return r;
}

__device__ __forceinline__ void fma2(unsigned long long& c, unsigned long long a, unsigned long long b) {
  asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(c) : "l"(a), "l"(b));
}

// grid.x: column tiles x cluster blocks (1 or 8), grid.y: row tiles, grid.z: products of a batch
template <int BM, bool CLUSTER>
__global__ void __launch_bounds__(TileShape<BM>::kThreads, TileShape<BM>::kBlocks)
gemm_f32_tiles_kernel(float* __restrict__ C, const float* __restrict__ A, const float* __restrict__ W, int M, int N, int K,
                      int lda, int ldw, int ldc, long long sa, long long sw, long long sc, int vec_a, int vec_w) {
  ccb::pdl_begin();
  using Sh = TileShape<BM>;
  constexpr int kTileThreads = Sh::kThreads;
  extern __shared__ __align__(16) float smem[];
  float* a_s = smem;                    // [2][kTileK][kPitch]
  float* w_s = smem + 2 * Sh::kA;       // [2][kTileK][kWPitch]
  float4* totals = reinterpret_cast<float4*>(smem + 2 * (Sh::kA + Sh::kW));   // [2 TM][threads]
  C += (size_t)blockIdx.z * sc;
  A += (size_t)blockIdx.z * sa;
  W += (size_t)blockIdx.z * sw;
  const int tid = threadIdx.x, ty = tid >> 4, tx = tid & 15;
  const int rank = CLUSTER ? blockIdx.x % kSegments : 0;
  const int n0 = (CLUSTER ? blockIdx.x / kSegments : blockIdx.x) * kTileN, m0 = blockIdx.y * BM;
  const int seg = segment_of(K);
  const int k_begin = rank * seg, k_end = min(K, CLUSTER ? k_begin + seg : K);
  constexpr int LA = BM * 4 / kTileThreads, LW = kTileN * 4 / kTileThreads;
  float4 ra[LA], rw[LW];

  auto piece = [&](const float* base, int ld, int row, int rows, int k, int vec) {
    float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
    if (row < rows) {
      const float* src = base + (size_t)row * ld + k;
      if (vec && k + 3 < k_end) {
        v = *reinterpret_cast<const float4*>(src);
      } else {
        if (k < k_end) v.x = src[0];
        if (k + 1 < k_end) v.y = src[1];
        if (k + 2 < k_end) v.z = src[2];
        if (k + 3 < k_end) v.w = src[3];
      }
    }
    return v;
  };
  auto load = [&](int k0) {
#pragma unroll
    for (int i = 0; i < LA; ++i) {
      const int idx = tid + kTileThreads * i;
      ra[i] = piece(A, lda, m0 + (idx >> 2), M, k0 + 4 * (idx & 3), vec_a);
    }
#pragma unroll
    for (int i = 0; i < LW; ++i) {
      const int idx = tid + kTileThreads * i;
      rw[i] = piece(W, ldw, n0 + (idx >> 2), N, k0 + 4 * (idx & 3), vec_w);
    }
  };
  auto store = [&](int st) {
    float* as = a_s + st * Sh::kA;
    float* ws = w_s + st * Sh::kW;
#pragma unroll
    for (int i = 0; i < LA; ++i) {
      const int idx = tid + kTileThreads * i, row = idx >> 2, k = 4 * (idx & 3);
      as[(k + 0) * Sh::kPitch + row] = ra[i].x;
      as[(k + 1) * Sh::kPitch + row] = ra[i].y;
      as[(k + 2) * Sh::kPitch + row] = ra[i].z;
      as[(k + 3) * Sh::kPitch + row] = ra[i].w;
    }
#pragma unroll
    for (int i = 0; i < LW; ++i) {
      const int idx = tid + kTileThreads * i, row = idx >> 2, k = 4 * (idx & 3);
      ws[(k + 0) * kWPitch + row] = rw[i].x;
      ws[(k + 1) * kWPitch + row] = rw[i].y;
      ws[(k + 2) * kWPitch + row] = rw[i].z;
      ws[(k + 3) * kWPitch + row] = rw[i].w;
    }
  };

  // columns tx * 4 .. + 3 (pairs 0, 1) and 64 + tx * 4 .. + 3 (pairs 2, 3) of rows ty * TM ..
  unsigned long long acc[TM][4];
#pragma unroll
  for (int i = 0; i < TM; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) acc[i][j] = 0ull;

  // the sums of the segment that has ended, into (or onto) the totals; a thread only touches its own places
  auto fold = [&](bool first) {
#pragma unroll
    for (int i = 0; i < TM; ++i)
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        float4& t = totals[(2 * i + h) * kTileThreads + tid];
        const float2 lo = *reinterpret_cast<const float2*>(&acc[i][2 * h]), hi = *reinterpret_cast<const float2*>(&acc[i][2 * h + 1]);
        float4 v = make_float4(lo.x, lo.y, hi.x, hi.y);
        if (!first) {
          const float4 o = t;
          v = make_float4(o.x + v.x, o.y + v.y, o.z + v.z, o.w + v.w);
        }
        t = v;
        acc[i][2 * h] = acc[i][2 * h + 1] = 0ull;
      }
  };

  bool first = true;
  int st = 0, left = seg;
  if (k_begin < k_end) {
    load(k_begin);
    store(0);
  }
  __syncthreads();
  for (int k0 = k_begin; k0 < k_end; k0 += kTileK) {
    const bool more = k0 + kTileK < k_end;
    if (more) load(k0 + kTileK);
    const float* as = a_s + st * Sh::kA + TM * ty;
    const float* ws = w_s + st * Sh::kW + 4 * tx;
#pragma unroll
    for (int k = 0; k < kTileK; ++k) {
      unsigned long long a[TM], b[4];
#pragma unroll
      for (int i = 0; i < TM; i += 4) {
        const float4 v = *reinterpret_cast<const float4*>(as + k * Sh::kPitch + i);
        a[i] = twice(v.x);
        a[i + 1] = twice(v.y);
        a[i + 2] = twice(v.z);
        a[i + 3] = twice(v.w);
      }
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const ulonglong2 v = *reinterpret_cast<const ulonglong2*>(ws + k * kWPitch + 64 * h);
        b[2 * h] = v.x;
        b[2 * h + 1] = v.y;
      }
#pragma unroll
      for (int i = 0; i < TM; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) fma2(acc[i][j], a[i], b[j]);
    }
    if (more) store(st ^ 1);
    __syncthreads();
    st ^= 1;
    left -= kTileK;
    if (left == 0 || !more) {
      fold(first);
      first = false;
      left = seg;
    }
  }
  if (CLUSTER && k_begin >= k_end) fold(true);   // a segment past K: zeros

  auto write = [&](int q, float4 v) {   // place q of this thread's: row q / 2, column half q % 2
    const int gm = m0 + ty * TM + (q >> 1), gn = n0 + (q & 1) * 64 + tx * 4;
    if (gm >= M) return;
    float* dst = C + (size_t)gm * ldc + gn;
    if (gn < N) dst[0] = v.x;
    if (gn + 1 < N) dst[1] = v.y;
    if (gn + 2 < N) dst[2] = v.z;
    if (gn + 3 < N) dst[3] = v.w;
  };
  if constexpr (CLUSTER) {
    namespace cg = cooperative_groups;
    const cg::cluster_group cluster = cg::this_cluster();
    cluster.sync();
    for (int q = rank; q < 2 * TM; q += kSegments) {
      float4 v = cluster.map_shared_rank(totals, 0)[q * kTileThreads + tid];
      float4 o[kSegments - 1];
#pragma unroll
      for (int s = 1; s < kSegments; ++s) o[s - 1] = cluster.map_shared_rank(totals, s)[q * kTileThreads + tid];
#pragma unroll
      for (int s = 0; s < kSegments - 1; ++s) v = make_float4(v.x + o[s].x, v.y + o[s].y, v.z + o[s].z, v.w + o[s].w);
      write(q, v);
    }
    cluster.sync();   // nobody leaves while its sums are read
  } else {
#pragma unroll
    for (int q = 0; q < 2 * TM; ++q) write(q, totals[q * kTileThreads + tid]);
  }
}

struct F32Product {
  float* C;
  const float *A, *W;
  int M, N, K, lda, ldw, ldc;
  long long sa, sw, sc;
  int batch;
};

template <int MR> int rows_go(const F32Product& p, int vec, cudaStream_t stream) {
  auto kernel = gemm_f32_rows_kernel<MR>;
  static std::atomic<unsigned long long> done{0};
  const int rc = ccb_allow_smem(kernel, RowsStage<MR>::kBytes, done);
  if (rc != 0) return rc;
  ccb_launch(kernel, dim3((p.N + kRowW - 1) / kRowW, 1, p.batch), kRowWarps * 32, RowsStage<MR>::kBytes, stream, p.C, p.A, p.W,
             p.M, p.N, p.K, p.lda, p.ldw, p.ldc, p.sa, p.sw, p.sc, vec);
  return ccb_launch_status();
}

template <int BM> int tiles_go(const F32Product& p, int vec_a, int vec_w, cudaStream_t stream) {
  const int gx = (p.N + kTileN - 1) / kTileN, gy = (p.M + BM - 1) / BM;
  // A block an SM computes as fast as two do (the multiply-adds are the bound), so tiles run in rounds of 148.  A
  // cluster's rounds are an eighth as long: it is taken where the tiles fill fewer than two rounds, and where a segment
  // is long enough to pay for the exchange.
  const long long tiles = (long long)gx * gy * p.batch;
  const bool cluster = tiles < 2 * 148 && p.K >= 512;
  constexpr int bytes = TileShape<BM>::kBytes;
  auto kernel = cluster ? gemm_f32_tiles_kernel<BM, true> : gemm_f32_tiles_kernel<BM, false>;
  static std::atomic<unsigned long long> done[2];
  const int rc = ccb_allow_smem(kernel, bytes, done[cluster]);
  if (rc != 0) return rc;
  if (cluster)
    ccb_launch_cluster(false, kSegments, kernel, dim3(gx * kSegments, gy, p.batch), TileShape<BM>::kThreads, bytes, stream, p.C, p.A, p.W,
                       p.M, p.N, p.K, p.lda, p.ldw, p.ldc, p.sa, p.sw, p.sc, vec_a, vec_w);
  else
    ccb_launch(kernel, dim3(gx, gy, p.batch), TileShape<BM>::kThreads, bytes, stream, p.C, p.A, p.W, p.M, p.N, p.K, p.lda, p.ldw, p.ldc,
               p.sa, p.sw, p.sc, vec_a, vec_w);
  return ccb_launch_status();
}

int gemm_f32_launch(const F32Product& p, cudaStream_t stream) {
  if (p.M <= 0 || p.N <= 0 || p.batch <= 0) return 0;
  if (p.K <= 0 || p.lda < p.K || p.ldw < p.K || p.ldc < p.N || p.batch > 65535) return CCB_REFUSE_SIZE;
  auto aligned = [](const float* x, int ld, long long stride) {   // rows of every product of the batch start on 16 bytes
    return ld % 4 == 0 && stride % 4 == 0 && (reinterpret_cast<uintptr_t>(x) & 15) == 0;
  };
  const int vec_a = aligned(p.A, p.lda, p.sa), vec_w = aligned(p.W, p.ldw, p.sw);
  if (p.M <= 2) return rows_go<2>(p, vec_a && vec_w, stream);
  if (p.M <= 4) return rows_go<4>(p, vec_a && vec_w, stream);
  if (p.M <= 8) return rows_go<8>(p, vec_a && vec_w, stream);
  if (p.M <= 16) return rows_go<16>(p, vec_a && vec_w, stream);
  if (p.M <= 32) return tiles_go<32>(p, vec_a, vec_w, stream);
  // tiles of 64 rows where 128 would leave more than an eighth of the rows empty that 64 does not
  const int r64 = (p.M + 63) / 64 * 64, r128 = (p.M + 127) / 128 * 128;
  if (8 * (r128 - r64) > r128) return tiles_go<64>(p, vec_a, vec_w, stream);
  return tiles_go<128>(p, vec_a, vec_w, stream);
}

}  // namespace

CCB_API int ccb_gemm_f32(float* C, const float* A, const float* W, int M, int N, int K, int lda, int ldw, int ldc,
                         cudaStream_t stream) {
  return gemm_f32_launch({C, A, W, M, N, K, lda, ldw, ldc, 0, 0, 0, 1}, stream);
}

// A batch of products of equal shapes at fixed strides (in elements): C_b = A_b W_b^T.
CCB_API int ccb_gemm_f32_batched(float* C, const float* A, const float* W, int M, int N, int K, int lda, int ldw,
                                 int ldc, long long sa, long long sw, long long sc, int batch, cudaStream_t stream) {
  return gemm_f32_launch({C, A, W, M, N, K, lda, ldw, ldc, sa, sw, sc, batch}, stream);
}
