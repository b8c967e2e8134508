// C = A * B^T in float32 on CUDA cores, for rows that can be read 16 bytes at a time: the products of the all-32-bit
// path.  Same forms and the same sums as gemm_simt.cu (groups of rows, gathered rows, gated epilogues; every output is
// one thread's sum over k in ascending order, so the results hold the same bits and a row's does not depend on how many
// other rows there are), with the operands brought by a ring of `cp.async` stages and read four k at a time.
//
// A tile is BM rows x BN features, k in steps of 32; a stage's rows lie in shared memory as they do in memory, 144 bytes
// apart, so that eight lanes' 16-byte reads of eight features meet no bank conflict and rows are broadcast.  What bounds
// a product depends on the rows that share a weight matrix, and so does the tile:
//   few rows        4 x 32, one warp: a stream of weights; many small CTAs keep enough bytes in flight even where a
//                   projection has few features.  Rows beyond four read the weights again, from L2: 20 rows of one
//                   matrix (6144 x 2048) 40 us, with the next tile 52; 33 rows 70 and 53.  Beside one another the groups
//                   fill the device by themselves: 4.3 rows a group 148 us and 204, 8.5 rows 228 and 212 (60 x 2048 x 1408).
//                   A matrix beyond L2 they read from memory: a head of 151936 x 2048 with 5 rows 431 us, with the next
//                   tile 320, 16 rows 843 and 328, 24 rows 1247 and 671 (4 rows 236 and 320); 32000 x 2048 with 5 rows 115
//                   and 88; half of 12288 x 4096 is still in L2: 8 rows 74 and 93, 12 rows 100 and 95
//                   Between, where 8 x 32 tiles of two warps are few (up to 400 CTAs), those: what counts there is the chain
//                   over k, and more CTAs beside one another (one matrix, rows x features x k: 16 x 6144 x 2048 29 us, with
//                   the tile before 33, with the next one 42; 32 x 2048 x 5632 50, 67, 108; 32 x 2048 x 2048 20, 28, 41; 768
//                   CTAs, 32 x 6144 x 2048: 65, 63, 48; 8 x 6144 x 2048 21, 23, 42); up to 24 rows not before the tile above is
//                   more than one CTA a SM (24 x 512 x 256 3.35 us, in 8 x 32 3.48; 8 x 2048 x 5632 42.1 and 43.0)
//   up to 64        16 x 64, two warps with 8 x 2 sums a thread (34 rows a group 472 us, with the next tile 518)
//   up to 128       32 x 64 with 4 x 4 sums a thread: 100 rows 112 us, with the tile before 152, with the one behind 140
//   more            64 x 64 with 8 x 4 sums a thread (gated 4 x 4), bound by the products themselves: 256 rows 184 us,
//                   32 x 64 210, 128 x 64 243; twice the CTAs of 128 x 64 leave less of the last round empty
// Requests of 257 tokens and four decoded ones through two layers of Qwen1.5-MoE-A2.7B's sizes: 36.0 -> 12.9 ms; three
// short ones through a model of width 256: 2.09 -> 1.43 ms.
#define NF_CHAIN_CLASS 0x40
#include "common.cuh"

namespace nf {
namespace {

constexpr size_t kGfL2 = 126u << 20, kGfFar = 230u << 20;    // bytes of a matrix: beyond L2; with next to nothing left in it
constexpr int kGfK = 32;                  // k a stage
constexpr int kGfRow = kGfK + 4;          // floats between two rows of a stage

// UNROLL: fours of k whose reads may be in flight together
template <int BM, int BN, int TM, int TN, int STAGES, bool GATED, int UNROLL = (BM > 16 ? 2 : 8)>
__global__ void __launch_bounds__((BM / TM) * (BN / TN), BM >= 64 ? 2 : 1)
gemm_f32_kernel(const float* __restrict__ A, int lda, const float* __restrict__ B, size_t b_group_stride,
                float* __restrict__ C, int ldc, int M, int N, int K, const int* __restrict__ offsets,
                const int* __restrict__ a_rows, int a_div, GatedActParams act) {
  constexpr int TX = BN / TN, NT = (BM / TM) * TX;
  constexpr int NCOL = GATED ? BN / 2 : BN;            // output columns a CTA (gated: gate rows, then their up rows)
  constexpr int PIECES = (BM + BN) * (kGfK / 4);       // 16-byte pieces of a stage
  extern __shared__ __align__(16) float gf_smem[];     // [STAGES][BM rows of A, BN rows of B][kGfRow]
  chain_wait(A, B, offsets, a_rows);
  const int g = blockIdx.z;
  const int row_begin = offsets ? offsets[g] : 0, row_end = offsets ? offsets[g + 1] : M;
  const int n0 = blockIdx.x * NCOL;
  const float* Bg = B + (size_t)g * b_group_stride;
  const int tx = threadIdx.x % TX, ty = threadIdx.x / TX;
  const int steps = (K + kGfK - 1) / kGfK;
  for (int m0 = row_begin + blockIdx.y * BM; m0 < row_end; m0 += gridDim.y * BM) {
    // this thread's pieces of a stage: where they come from (null: zeros) and where they go
    constexpr int MINE = (PIECES + NT - 1) / NT;
    const float* src[MINE];
#pragma unroll
    for (int i = 0; i < MINE; ++i) {
      const int x = threadIdx.x + i * NT, r = x / (kGfK / 4);
      src[i] = nullptr;
      if (r < BM) {
        const int row = m0 + r;
        if (row < row_end) src[i] = A + (size_t)(a_rows ? a_rows[row] / a_div : row) * lda;
      } else if (r < BM + BN) {
        const int f = r - BM, c = n0 + (GATED ? f % NCOL : f);
        if (c < N) src[i] = Bg + (size_t)(GATED && f >= NCOL ? N + c : c) * K;
      }
    }
    auto fetch = [&](int step) {
      if (step < steps) {
        float* st = gf_smem + (size_t)(step % STAGES) * (BM + BN) * kGfRow;
#pragma unroll
        for (int i = 0; i < MINE; ++i) {
          const int x = threadIdx.x + i * NT;
          if (PIECES % NT == 0 || x < PIECES) {
            const int r = x / (kGfK / 4), k = step * kGfK + (x % (kGfK / 4)) * 4;
            const bool ok = src[i] != nullptr && k < K;
            cp16_or_zeros(st + r * kGfRow + (x % (kGfK / 4)) * 4, ok ? src[i] + k : A, ok);
          }
        }
      }
      asm volatile("cp.async.commit_group;" ::: "memory");
    };
    float acc[TM][TN];
#pragma unroll
    for (int i = 0; i < TM; ++i)
#pragma unroll
      for (int j = 0; j < TN; ++j) acc[i][j] = 0.f;
#pragma unroll
    for (int s = 0; s < STAGES - 1; ++s) fetch(s);
    for (int step = 0; step < steps; ++step) {
      asm volatile("cp.async.wait_group %0;" ::"n"(STAGES - 2) : "memory");
      __syncthreads();                    // the stage is in, and everyone is done with the one that is filled next
      fetch(step + STAGES - 1);
      const float* as = gf_smem + (size_t)(step % STAGES) * (BM + BN) * kGfRow + ty * TM * kGfRow;
      const float* bs = gf_smem + (size_t)(step % STAGES) * (BM + BN) * kGfRow + (BM + tx) * kGfRow;
#pragma unroll UNROLL
      for (int k = 0; k < kGfK; k += 4) {
        float a[TM][4], b[TN][4];
#pragma unroll
        for (int i = 0; i < TM; ++i) load4(as + i * kGfRow + k, a[i]);
#pragma unroll
        for (int j = 0; j < TN; ++j) load4(bs + j * TX * kGfRow + k, b[j]);
#pragma unroll
        for (int e = 0; e < 4; ++e)
#pragma unroll
          for (int i = 0; i < TM; ++i)
#pragma unroll
            for (int j = 0; j < TN; ++j) acc[i][j] = fmaf(a[i][e], b[j][e], acc[i][j]);
      }
    }
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    __syncthreads();                      // the ring is free for the next rows
#pragma unroll
    for (int i = 0; i < TM; ++i) {
      const int r = m0 + ty * TM + i;
      if (r >= row_end) continue;
      if (GATED) {
#pragma unroll
        for (int j = 0; j < TN / 2; ++j) {
          const int c = n0 + tx + TX * j;
          if (c < N) C[(size_t)r * ldc + c] = gated_act(acc[i][j], acc[i][j + TN / 2], act);
        }
      } else {
#pragma unroll
        for (int j = 0; j < TN; ++j) {
          const int c = n0 + tx + TX * j;
          if (c < N) C[(size_t)r * ldc + c] = act.kind == kActRelu2 ? relu_square(acc[i][j]) : acc[i][j];
        }
      }
    }
  }
}

struct GfCall {
  const float *A, *B;
  float* C;
  int lda, ldc, M, N, K, groups, max_rows;
  size_t bgs;
  const int *offsets, *a_rows;
  int a_div;
  GatedActParams act;
};

template <int BM, int BN, int TM, int TN, int STAGES, bool GATED>
int gf_launch(const GfCall& c, int row_tiles, cudaStream_t stream) {
  constexpr int NCOL = GATED ? BN / 2 : BN;
  constexpr size_t smem = (size_t)STAGES * (BM + BN) * kGfRow * sizeof(float);
  static bool set = false;
  if (!set) {
    cudaError_t e = cudaFuncSetAttribute(gemm_f32_kernel<BM, BN, TM, TN, STAGES, GATED>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    NF_REQUIRE(e == cudaSuccess, "gemm: cannot have %zu bytes of shared memory: %s", smem, cudaGetErrorString(e));
    set = true;
  }
  launch_chained(gemm_f32_kernel<BM, BN, TM, TN, STAGES, GATED>, dim3((c.N + NCOL - 1) / NCOL, row_tiles, c.groups),
                 dim3((BM / TM) * (BN / TN)), smem, stream, c.A, c.lda, c.B, c.bgs, c.C, c.ldc, c.M, c.N, c.K, c.offsets, c.a_rows,
                 c.a_div, c.act);
  return check_launch("gemm_f32");
}

template <bool GATED>
int gf_dispatch(const GfCall& c, cudaStream_t stream) {
  // rows a weight matrix meets: a group's on average (its CTAs walk on where it has more)
  const int rows = c.groups > 1 ? (c.M + c.groups - 1) / c.groups : c.M;
  auto tiles = [&](int bm) {
    const int most = (c.max_rows + bm - 1) / bm, usual = (2 * rows + bm - 1) / bm;
    const int n = c.groups > 1 && usual < most ? usual : most;
    return n < 65535 ? n : 65535;
  };
  // (the lines lie between the measured sizes at which the tile below and the one above were the faster)
  const bool alone = c.groups == 1;
  const size_t matrix = (size_t)c.N * (GATED ? 2 : 1) * c.K * sizeof(float);
  if constexpr (!GATED)
    if (alone && rows > 4 && rows <= 32 && (c.N + 31) / 32 * ((c.max_rows + 7) / 8) <= 400 && matrix <= kGfL2 &&
        (rows > 24 || (c.N + 31) / 32 * ((c.max_rows + 3) / 4) > 148))      // up to one CTA a SM of the tile below: that one
      return gf_launch<8, 32, 4, 1, 8, false>(c, tiles(8), stream);
  if (rows <= (!alone ? 5 : matrix > kGfFar ? 4 : matrix > kGfL2 ? 10 : 24)) return gf_launch<4, GATED ? 64 : 32, 4, GATED ? 2 : 1, 6, GATED>(c, tiles(4), stream);
  if (rows <= 64) return gf_launch<16, 64, 8, 2, 4, GATED>(c, tiles(16), stream);
  if (rows <= 128) return gf_launch<32, 64, 4, 4, 4, GATED>(c, tiles(32), stream);
  if (GATED) return gf_launch<64, 64, 4, 4, 3, GATED>(c, tiles(64), stream);
  return gf_launch<64, 64, 8, 4, 3, GATED>(c, tiles(64), stream);
}

}  // namespace

bool gemm_f32_takes(const void* A, int lda, const void* B, size_t bgs, int K) {
  return K % 4 == 0 && lda % 4 == 0 && bgs % 4 == 0 && (uintptr_t)A % 16 == 0 && (uintptr_t)B % 16 == 0;
}

int gemm_f32(const void* A, int lda, const void* B, size_t bgs, void* C, int ldc, int M, int N, int K, int groups, int max_rows,
             const int* offsets, const int* a_rows, int a_div, bool gated, GatedActParams act, cudaStream_t stream) {
  NF_REQUIRE(groups <= 65535, "gemm: too many groups (%d)", groups);
  const GfCall c{(const float*)A, (const float*)B, (float*)C, lda, ldc, M, N, K, groups, max_rows, bgs, offsets, a_rows, a_div, act};
  return gated ? gf_dispatch<true>(c, stream) : gf_dispatch<false>(c, stream);
}

}  // namespace nf
