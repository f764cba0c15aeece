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
//   tiles  M > 16: tiles of 12 to 128 rows x 128 columns, two multiply-adds an instruction (fma.rn.f32x2); `choose_tiles`
//          picks their height, so that few rows of a tile are empty and few SMs idle in the last round.  Where the tiles do
//          not fill the machine a cluster of eight blocks takes a tile, a segment each, and adds up through distributed
//          shared memory.
// What bounds them: the rows kernel the stream of W (2 x 16,384 x 2,048: 34 us, 3.9 TB/s; 2 x 32,000 x 2,048: 57 us, 4.6
// TB/s) until many rows make it the reads of A (16 x 16,384 x 2,048: 66 us); the tiles kernel the multiply-adds, of which
// registers alone reach 65 TFLOP/s, with reads of shared memory beside them.  us, tiles of 32, 64 or 128 rows with 8 x 8 places
// a thread, one block an SM / so: 17 x 16,384 x 2,048 77 / 60, 64 x 4,096 x 2,048 35 / 35, 100 x 16,384 x 2,048 267 / 187,
// 210 x 2,048 x 8,192 307 / 174, 210 x 16,384 x 2,048 524 / 349 (40 TFLOP/s), 300 x 16,384 x 2,048 511 / 501, 2,048 x 4,096 x
// 4,096 1,593 / 1,389 (49).  Sums of even and of odd k side by side (no element stored by itself, eight columns a thread) took
// 419 us for 210 x 16,384 x 2,048.
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
// A block: a tile of WR x WC warps, 128 columns; a thread TM rows x TN columns, two columns a multiply-add.  What it reads from
// shared memory comes back at 128 bytes a cycle and SM whether lanes read the same or not, so TM + TN cycles a k and warp stand
// against TM TN / 4 of multiply-adds: sixteen columns a thread where there are rows enough for four warps below one another
// (eight left the reads the bound), eight and warps side by side for fewer rows.  Several blocks an SM: one's first loads and
// last exchange run under another's multiply-adds.
constexpr int kTileK = 16;
constexpr int kTileN = 128;
constexpr int kTilePitch = kTileN + 4;   // floats from k to k
constexpr int kTileMinRows = 3, kTileMaxRows = 8;   // TM

template <int TM_, int TN_, int WR_, int WC_> struct TileShape {
  static constexpr int TM = TM_, TN = TN_, WR = WR_, WC = WC_;
  static_assert(WC * 8 * TN == kTileN, "128 columns");
  static constexpr int kThreads = 32 * WR * WC;
  static constexpr int kBlocks = TN == 16 ? 2 : WR == 2 ? 3 : 5;   // an SM
  static constexpr int kWarpRows = 4 * TM, kRows = WR * kWarpRows;
  static constexpr int kPlaces = TM > 4 ? 32 : 16;                 // of a warp's rows in shared memory
  static constexpr int kPitchA = WR * kPlaces + 4;
  static constexpr int kStage = kTileK * (kPitchA + kTilePitch);   // floats
  static constexpr int kTotals = kRows * kTileN;                   // a segment's tile, or the total so far
  static constexpr int kQuads = TM * TN / 4;                       // fours of sums a thread has
  // where a warp's row lies: four to a lane's quarter first, then the quarter's others from place 16 on
  static __device__ __forceinline__ int place(int row) {
    constexpr int kFirst = TM < 4 ? TM : 4, kRest = TM > 4 ? TM - 4 : 1;
    if (row < 4 * kFirst) return row / kFirst * 4 + row % kFirst;
    return 16 + (row - 16) / kRest * 4 + (row - 16) % kRest;
  }
  static constexpr int bytes(bool cluster) {   // (a cluster's block has one segment: its sums take the stages' place)
    return 4 * (cluster ? (2 * kStage > kTotals ? 2 * kStage : kTotals) : 2 * kStage + kTotals);
  }
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
template <class Sh, bool CLUSTER>
__global__ void __launch_bounds__(Sh::kThreads, Sh::kBlocks)
gemm_f32_tiles_kernel(float* __restrict__ C, const float* __restrict__ A, const float* __restrict__ W, int M, int N, int K,
                      int lda, int ldw, int ldc, long long sa, long long sw, long long sc, int vec_a, int vec_w) {
  ccb::pdl_begin();
  constexpr int TM = Sh::TM, TN = Sh::TN, kThreads = Sh::kThreads;
  extern __shared__ __align__(16) float smem[];
  float4* totals = reinterpret_cast<float4*>(smem + (CLUSTER ? 0 : 2 * Sh::kStage));   // [kQuads][threads]
  C += (size_t)blockIdx.z * sc;
  A += (size_t)blockIdx.z * sa;
  W += (size_t)blockIdx.z * sw;
  const int tid = threadIdx.x, wr = (tid >> 5) % Sh::WR, wc = (tid >> 5) / Sh::WR, ty = (tid >> 3) & 3, tx = tid & 7;
  const int rank = CLUSTER ? blockIdx.x % kSegments : 0;
  const int n0 = (CLUSTER ? blockIdx.x / kSegments : blockIdx.x) * kTileN, m0 = blockIdx.y * Sh::kRows;
  const int seg = segment_of(K);
  const int k_begin = rank * seg, k_end = min(K, CLUSTER ? k_begin + seg : K);
  const int steps = k_begin < k_end ? (k_end - k_begin + kTileK - 1) / kTileK : 0;

  // A thread takes four k of some rows, to registers and from there to shared memory; for the second eight k the rows lie
  // with eights exchanged, so that a warp's stores fall into different banks.
  const int q4 = 4 * (tid & 3), cr = tid >> 2, flip = q4 & 8;
  constexpr int kPass = kThreads / 4, LA = (Sh::kRows + kPass - 1) / kPass, LW = kTileN / kPass;
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
  auto load = [&](int step) {
    const int k = k_begin + step * kTileK + q4;
#pragma unroll
    for (int i = 0; i < LA; ++i)
      if (Sh::kRows % kPass == 0 || cr + kPass * i < Sh::kRows) ra[i] = piece(A, lda, m0 + cr + kPass * i, M, k, vec_a);
#pragma unroll
    for (int i = 0; i < LW; ++i) rw[i] = piece(W, ldw, n0 + cr + kPass * i, N, k, vec_w);
  };
  auto put = [&](float* to, int pitch, float4 v) {
    to[0] = v.x;
    to[pitch] = v.y;
    to[2 * pitch] = v.z;
    to[3 * pitch] = v.w;
  };
  auto store = [&](int step) {
    float* a_s = smem + (step & 1) * Sh::kStage + q4 * Sh::kPitchA;
    float* w_s = smem + (step & 1) * Sh::kStage + kTileK * Sh::kPitchA + q4 * kTilePitch;
#pragma unroll
    for (int i = 0; i < LA; ++i) {
      const int row = cr + kPass * i;
      if (Sh::kRows % kPass == 0 || row < Sh::kRows)
        put(a_s + row / Sh::kWarpRows * Sh::kPlaces + (Sh::place(row % Sh::kWarpRows) ^ flip), Sh::kPitchA, ra[i]);
    }
#pragma unroll
    for (int i = 0; i < LW; ++i) put(w_s + ((cr + kPass * i) ^ flip), kTilePitch, rw[i]);
  };

  // columns col0 + 32 j .. + 3 (pairs 2 j, 2 j + 1)
  const int col0 = wc * 8 * TN + 4 * tx;
  unsigned long long acc[TM][TN / 2];
#pragma unroll
  for (int i = 0; i < TM; ++i)
#pragma unroll
    for (int j = 0; j < TN / 2; ++j) acc[i][j] = 0ull;

  // the sums of the segment that has ended, into (or onto) the totals; a thread only touches its own places
  auto fold = [&](bool first) {
#pragma unroll
    for (int i = 0; i < TM; ++i)
#pragma unroll
      for (int j = 0; j < TN / 4; ++j) {
        float4& t = totals[(TN / 4 * i + j) * kThreads + tid];
        const float2 lo = *reinterpret_cast<const float2*>(&acc[i][2 * j]), hi = *reinterpret_cast<const float2*>(&acc[i][2 * j + 1]);
        float4 v = make_float4(lo.x, lo.y, hi.x, hi.y);
        if (!first) {
          const float4 o = t;
          v = make_float4(o.x + v.x, o.y + v.y, o.z + v.z, o.w + v.w);
        }
        t = v;
        acc[i][2 * j] = acc[i][2 * j + 1] = 0ull;
      }
  };

  if (steps > 0) {
    load(0);
    store(0);
  }
  __syncthreads();
  bool first = true;
  int left = seg;
  for (int step = 0; step < steps; ++step) {
    if (step + 1 < steps) load(step + 1);
    const float* stage = smem + (step & 1) * Sh::kStage;
#pragma unroll
    for (int k = 0; k < kTileK; ++k) {
      const float* a_s = stage + wr * Sh::kPlaces + ((4 * ty) ^ (k & 8)) + k * Sh::kPitchA;
      const float* w_s = stage + kTileK * Sh::kPitchA + (col0 ^ (k & 8)) + k * kTilePitch;
      unsigned long long b[TN / 2];
#pragma unroll
      for (int j = 0; j < TN / 4; ++j) {
        const ulonglong2 v = *reinterpret_cast<const ulonglong2*>(w_s + 32 * j);
        b[2 * j] = v.x;
        b[2 * j + 1] = v.y;
      }
#pragma unroll
      for (int g = 0; g < (TM + 3) / 4; ++g) {
        const float4 v = *reinterpret_cast<const float4*>(a_s + 16 * g);
        const float x[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
        for (int i = 4 * g; i < TM && i < 4 * g + 4; ++i) {
          const unsigned long long a = twice(x[i & 3]);
#pragma unroll
          for (int j = 0; j < TN / 2; ++j) fma2(acc[i][j], a, b[j]);
        }
      }
    }
    if (step + 1 < steps) store(step + 1);
    __syncthreads();   // the next stage is there, and everybody has read this one
    left -= kTileK;
    if (left == 0 || step + 1 == steps) {
      fold(first);
      first = false;
      left = seg;
    }
  }
  if (CLUSTER && steps == 0) fold(true);   // a segment past K: zeros

  auto write = [&](int q, float4 v) {   // the thread's four q: a row, four neighbouring columns
    const int i = q / (TN / 4), row = i < 4 ? ty * (TM < 4 ? TM : 4) + i : 16 + ty * (TM - 4) + (i - 4);
    const int gm = m0 + wr * Sh::kWarpRows + row, gn = n0 + col0 + 32 * (q % (TN / 4));
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
    for (int q = rank; q < Sh::kQuads; q += kSegments) {
      float4 v = cluster.map_shared_rank(totals, 0)[q * kThreads + tid];
      float4 o[kSegments - 1];
#pragma unroll
      for (int s = 1; s < kSegments; ++s) o[s - 1] = cluster.map_shared_rank(totals, s)[q * kThreads + tid];
#pragma unroll
      for (int s = 0; s < kSegments - 1; ++s) v = make_float4(v.x + o[s].x, v.y + o[s].y, v.z + o[s].z, v.w + o[s].w);
      write(q, v);
    }
    cluster.sync();   // nobody leaves while its sums are read
  } else {
#pragma unroll
    for (int q = 0; q < Sh::kQuads; ++q) write(q, totals[q * kThreads + tid]);
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

template <class Sh> int tiles_go(const F32Product& p, int vec_a, int vec_w, bool cluster, cudaStream_t stream) {
  const int bytes = Sh::bytes(cluster);
  const int gx = (p.N + kTileN - 1) / kTileN, gy = (p.M + Sh::kRows - 1) / Sh::kRows;
  auto kernel = cluster ? gemm_f32_tiles_kernel<Sh, true> : gemm_f32_tiles_kernel<Sh, false>;
  static std::atomic<unsigned long long> done[2];
  const int rc = ccb_allow_smem(kernel, bytes, done[cluster]);
  if (rc != 0) return rc;
  if (cluster)
    ccb_launch_cluster(false, kSegments, kernel, dim3(gx * kSegments, gy, p.batch), Sh::kThreads, bytes, stream, p.C, p.A, p.W,
                       p.M, p.N, p.K, p.lda, p.ldw, p.ldc, p.sa, p.sw, p.sc, vec_a, vec_w);
  else
    ccb_launch(kernel, dim3(gx, gy, p.batch), Sh::kThreads, bytes, stream, p.C, p.A, p.W, p.M, p.N, p.K, p.lda, p.ldw, p.ldc,
               p.sa, p.sw, p.sc, vec_a, vec_w);
  return ccb_launch_status();
}

// The rows of a tile and whether a cluster shares it, by the cycles that the busiest SM would need: its blocks go round by
// round, a k of a block costs an SM its multiply-adds or its reads of shared memory, whichever is more, and stores beside them;
// a round is no less than one thread's chain of instructions, under which only a tenth of what other blocks do hides; a block
// multiplies some 10 k more than it has.  How many clusters of eight find room with so many blocks on an SM is kRoom (what
// cudaOccupancyMaxActiveClusters says here: the 16th gives some SM a second block, and takes as long as 33).  The constants are
// fitted to 390 shapes of 17 to 2,048 rows, each timed with every tile: what is chosen takes 1 per cent longer than the best on
// average (32 and 8 of 390 more than 5 and 10).  With 136 SMs for clusters and one block's work hidden under another's chain, 37 of
// 353 other shapes took more than 2 per cent longer than with tiles of 32, 64 and 128 rows alone, 29 more than 5; now 10 and 3 (us, such tiles /
// then / now: 55 x 655 x 1,086 twice 15.6 / 23.0 / 15.4, 59 x 1,536 x 12,224 101 / 136 / 106, 285 x 365 x 12,978 119 / 159 / 134; all
// 353 on average 1 / 0.70 / 0.67).
constexpr int kRoom[] = {0, 15, 33, 48, 71, 86};
struct TileChoice {
  int family, tm;   // family 0: 16 columns a thread, 4 x 1 warps; 1: 8, 2 x 2; 2: 8, 1 x 2
  bool cluster;
};
TileChoice choose_tiles(int M, int N, int K, int batch) {
  TileChoice best{0, kTileMaxRows, false};
  double least = 0;
  for (int family = 0; family < 3; ++family) {
    const int tn = family == 0 ? 16 : 8, wr = 4 >> family, warps = family == 2 ? 2 : 4, blocks = family == 0 ? 2 : family == 1 ? 3 : 5;
    for (int tm = kTileMaxRows; tm >= (family == 0 ? kTileMinRows + 1 : kTileMinRows); --tm) {   // (three rows of sixteen columns: never the best)
      const int rows = 4 * wr * tm;
      const double adds = warps * tm * tn / 4., reads = 1.4 * warps * tn, cost = (adds > reads ? adds : reads) + 11, chain = 1.2 * tm * tn + 33;
      const auto round = [&](int n) {   // of n blocks an SM
        const double hidden = chain + .9 * (n - 1) * cost;
        return n == 0 ? 0. : n * cost > hidden ? n * cost : hidden;
      };
      const long long tiles = (long long)((N + kTileN - 1) / kTileN) * ((M + rows - 1) / rows) * batch;
      for (int cluster = 0; cluster < 2; ++cluster) {   // (units: blocks, or clusters of eight)
        const int full = cluster ? kRoom[blocks] : 148 * blocks, left = (int)(tiles % full);
        int rest = cluster ? 0 : (left + 147) / 148;
        while (cluster && kRoom[rest] < left) ++rest;
        const double k = (cluster ? segment_of(K) : K) + 10;
        const double cycles = (tiles / full * round(blocks) + round(rest)) * k + (cluster ? 2400 : 0);
        if (least == 0 || cycles < least) least = cycles, best = {family, tm, cluster != 0};
      }
    }
  }
  return best;
}

template <int TM> int tiles_of(const F32Product& p, int vec_a, int vec_w, const TileChoice& t, cudaStream_t stream) {
  if constexpr (TM > kTileMinRows)
    if (t.family == 0) return tiles_go<TileShape<TM, 16, 4, 1>>(p, vec_a, vec_w, t.cluster, stream);
  if (t.family == 1) return tiles_go<TileShape<TM, 8, 2, 2>>(p, vec_a, vec_w, t.cluster, stream);
  return tiles_go<TileShape<TM, 8, 1, 2>>(p, vec_a, vec_w, t.cluster, stream);
}

int tiles_any(const F32Product& p, int vec_a, int vec_w, const TileChoice& t, cudaStream_t stream) {
  switch (t.tm) {
    case 3: return tiles_of<3>(p, vec_a, vec_w, t, stream);
    case 4: return tiles_of<4>(p, vec_a, vec_w, t, stream);
    case 5: return tiles_of<5>(p, vec_a, vec_w, t, stream);
    case 6: return tiles_of<6>(p, vec_a, vec_w, t, stream);
    case 7: return tiles_of<7>(p, vec_a, vec_w, t, stream);
    default: return tiles_of<8>(p, vec_a, vec_w, t, stream);
  }
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
  constexpr int kMost = 65535 * 4 * kTileMinRows;   // rows of a launch, whatever the tile's height
  for (F32Product q = p;; q.M -= kMost, q.A += (size_t)kMost * q.lda, q.C += (size_t)kMost * q.ldc) {
    F32Product part = q;
    part.M = q.M < kMost ? q.M : kMost;
    const int rc = tiles_any(part, vec_a, vec_w, choose_tiles(part.M, part.N, part.K, part.batch), stream);
    if (rc != 0 || q.M <= kMost) return rc;
  }
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
