// Causal grouped-query attention over the paged cache in float32: the all-32-bit path's, with the options and the
// mathematics of paged_attention_generic_kernel (attention_generic.cu).  Scores are one chain of products
// over the head size, keys are taken in blocks of 32 that begin at multiples of 32, in ascending order, and a block's
// values are added one key after the other; so a row's bits depend on its own position alone, however the step was cut,
// and are the same in every form below.  (The other kernel's blocks begin at a window's first key, and the kept first
// keys are a run of their own there: the same bits in both where no window passes a key, roundings apart where one does.)
//
// What bounds it: nothing but the way the keys reach the multiply-add units.  With one warp a row and head, every row
// fetched all keys for itself, 32 lanes from 32 rows of memory: 308 us for 256 rows of 16 heads of 128 over 257 keys
// (0.27 GFLOP, 4 us at the pipes' rate), now 49; four single rows over 257 keys 139, now 18.  Here a CTA takes up to 8
// queries that see the same keys (rows of a segment times the heads of a key head; 16 with more than 8 heads a key head),
// and brings 32, 64 or 128 keys and values to shared memory once for all of them, the next keys while the softmax and the
// values are worked on, the next values while the scores are.
//   scores   a lane a key, a warp a block of 32 keys and a share of the queries: a 16-byte piece of the key's row
//            against the same piece of each query's (a broadcast); rows lie D + 4 floats apart, so that eight lanes'
//            pieces meet no bank conflict
//   softmax  a warp a query, its blocks one after the other
//   values   a thread a dimension (two for heads beyond 128), every query's sum in a register
// Steps of single rows take forms of 1, 2 or 4 queries.  With few CTAs the chain from key to key is what counts, and four
// blocks at a time are the fastest; but that is one CTA a SM at heads of 128, and more CTAs come in rounds: the form is
// the one of most blocks whose CTAs all find room (af_blocks).  A tile whose keys are one block has all warps fetch and
// score it.  us, heads of 128, four blocks at a time always / now / one warp a row and head (attention_generic.cu):
//   64 rows of 16 heads (16 key heads)    8 keys 52.4 / 10.4 / 9.7,  100 69 / 30 / 115,   1,024 330 / 245 / 1,197
//   32 rows of 16 heads                   8 keys 29.9 / 5.7 / 9.4,   100 35 / 16 / 59,    1,024 188 / 105 / 1,205
//   4 rows of 16 heads                    8 keys 8.1 / 5.1 / 9.0,    100 9.4 / 9.3 / 57,  1,024 46 / 47 / 582
//   4 rows of 28 heads (4 key heads)      8 keys 13.2 / 5.7 / 9.2,   100 28 / 14 / 58,    1,024 192 / 97 / 537
//   256 rows of 28 heads                  257 keys 142 / 67 / 246;   96 rows of 32 prompts of 2 and 4 tokens 19.8 / 8.8 / 8.6
// Where it is still behind one warp a row: more than 888 CTAs (six a SM) of requests of fewer than ten tokens.
#define NF_CHAIN_CLASS 8
#include "common.cuh"

namespace nf {
namespace {

constexpr int kAfThreads = 128;

struct AfArgs {
  const float* qkv;
  const float* pages;
  const int *block_table, *positions, *row_seg, *seg_row0;
  float* out;
  const float *slopes, *gate, *sig_bias;
  int q_row_stride, bt_width, T, S, Hq, Hkv, D, page_size, num_pages, window, keep_first, gate_ld;
  int heads_tile, rows_tile, head_tiles;       // queries of a CTA: heads of a key head x rows; CTAs a key head
  float scale, softcap;
};

__device__ __forceinline__ void af_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N> __device__ __forceinline__ void af_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

// Q queries, KB blocks of 32 keys at a time
template <int Q, int KB>
constexpr size_t af_floats(int D) {
  return (size_t)KB * 32 * (D + 4) + (size_t)KB * 32 * D + (size_t)Q * D + (size_t)Q * KB * 32 + (size_t)Q * KB;
}

// What a CTA works on: rows row0.. of one segment, `heads` query heads of a key head from head0 on.  Query x: row
// row0 + x / heads, head head0 + x % heads.
struct AfTile {
  const int* bt;
  int row0, rows, head0, heads, kvh, pos_most, pos_least;
};

// DP: the head size rounded up (32, 64, 128, 256)
template <int Q, int KB, int DP>
__device__ __forceinline__ void af_tile(const AfArgs& a, const AfTile& t, float* af_smem, int* q_pos, int* q_lo, float* q_slope) {
  constexpr int NW = kAfThreads / 32;
  constexpr int KT = KB * 32;                               // keys at a time
  constexpr int SHARES = NW / KB;                           // warps that share a block of keys, each with its queries
  constexpr int QS = Q >= SHARES ? Q / SHARES : 1;          // queries a warp scores
  constexpr int DI = DP > kAfThreads ? DP / kAfThreads : 1; // dimensions a thread
  constexpr int GROUPS = DP < kAfThreads ? kAfThreads / DP : 1;    // threads that share a dimension, each with its queries
  constexpr int QV = Q >= GROUPS ? Q / GROUPS : 1;          // queries a thread adds up
  constexpr int QW = (Q + NW - 1) / NW;                     // queries whose softmax a warp keeps
  constexpr int RW = KT / NW;                               // key rows a warp fetches
  constexpr int LR = DP / 4 < 32 ? DP / 4 : 32;             // lanes a row
  const int D = a.D, DK = D + 4;
  float* const ks = af_smem;                                // [KT][D + 4]
  float* const vs = ks + (size_t)KT * DK;                   // [KT][D]
  float* const qs = vs + (size_t)KT * D;                    // [Q][D]
  float* const ps = qs + (size_t)Q * D;                     // [Q][KT] scores, then weights; a weight below 0: not seen
  float* const as = ps + (size_t)Q * KT;                    // [KB][Q] what a block scales the sums before it by
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int row0 = t.row0, head0 = t.head0, heads = t.heads, nq = t.rows * t.heads, pos_most = t.pos_most, pos_least = t.pos_least;
  const int* const bt = t.bt;
  const size_t head_stride = (size_t)a.page_size * D, page_stride = (size_t)2 * a.Hkv * head_stride;
  const float* const kv_head = a.pages + (size_t)t.kvh * head_stride;

  for (int x = warp; x < nq; x += NW) {
    const float* q = a.qkv + (size_t)(row0 + x / heads) * a.q_row_stride + (size_t)(head0 + x % heads) * D;
    for (int d = lane; d < D; d += 32) qs[x * D + d] = q[d];
  }
  if (tid < nq) {
    const int p = a.positions[row0 + tid / heads];
    q_pos[tid] = p;
    q_lo[tid] = a.window > 0 ? max(0, p - a.window + 1) : 0;
    q_slope[tid] = a.slopes ? a.slopes[head0 + tid % heads] : 0.f;
  }
  const int lo_least = a.window > 0 ? max(0, pos_least - a.window + 1) : 0;
  const int lo_most = a.window > 0 ? max(0, pos_most - a.window + 1) : 0;
  // the keys' steps: those of the kept first keys, then from the first window's begin on
  const int kept = min(a.keep_first, lo_most);              // keys below this one are seen without the window
  const int step_lo = lo_least / KT, kept_steps = min(step_lo, (kept + KT - 1) / KT);
  const int steps = kept_steps + (pos_most / KT + 1 - step_lo);
  auto first_key = [&](int step) { return (step < kept_steps ? step : step_lo + step - kept_steps) * KT; };

  auto key_row = [&](int j) -> const float* {
    const int lp = j / a.page_size, page = lp < a.bt_width ? bt[lp] : -1;
    return page >= 0 && page < a.num_pages ? kv_head + (size_t)page * page_stride + (size_t)(j % a.page_size) * D : nullptr;
  };
  // lane r keeps where row r of the warp's share of a step's keys lies (null: zeros in its place)
  auto my_row = [&](int step) -> const float* {
    const int j = first_key(step) + warp * RW + lane;
    return step < steps && lane < RW && j <= pos_most ? key_row(j) : nullptr;
  };
  auto fetch = [&](const float* mine, float* dst, int ld, size_t off) {
    const int c0 = (lane % LR) * 4;
#pragma unroll 8
    for (int r0 = 0; r0 < RW; r0 += 32 / LR) {
      const int r = r0 + lane / LR;
      const float* src = reinterpret_cast<const float*>(__shfl_sync(0xffffffffu, reinterpret_cast<unsigned long long>(mine), r));
#pragma unroll
      for (int c = c0; c < DP; c += LR * 4)
        if (c < D) cp16_or_zeros(dst + (size_t)(warp * RW + r) * ld + c, src ? src + off + c : a.pages, src != nullptr);
    }
    af_commit();
  };

  float m[QW], l[QW];
#pragma unroll
  for (int i = 0; i < QW; ++i) m[i] = -INFINITY, l[i] = 0.f;
  float acc[DI][QV];
#pragma unroll
  for (int i = 0; i < DI; ++i)
#pragma unroll
    for (int x = 0; x < QV; ++x) acc[i][x] = 0.f;
  const int vd = tid % DP, vq0 = DP < kAfThreads ? (tid / DP) * QV : 0;       // this thread's dimension and first query
  const int sb = warp % KB, sq0 = (warp / KB) * QS;                          // this warp's block and first query

  const float* mine = my_row(0);
  fetch(mine, ks, DK, 0);
  fetch(mine, vs, D, (size_t)a.Hkv * head_stride);
  for (int step = 0; step < steps; ++step) {
    const int j0 = first_key(step);
    af_wait<1>();                                           // the keys are in
    __syncthreads();
    if (sq0 < nq) {
      float s[QS];
#pragma unroll
      for (int x = 0; x < QS; ++x) s[x] = 0.f;
      const float* k = ks + (size_t)(sb * 32 + lane) * DK;
      const float* q = qs + (size_t)sq0 * D;
      if (j0 + sb * 32 <= pos_most) {
#pragma unroll 4
        for (int d = 0; d < D; d += 4) {
          float kk[4];
          load4(k + d, kk);
#pragma unroll
          for (int x = 0; x < QS; ++x) {
            float qq[4];
            load4(q + x * D + d, qq);
#pragma unroll
            for (int e = 0; e < 4; ++e) s[x] = fmaf(qq[e], kk[e], s[x]);
          }
        }
      }
      const int j = j0 + sb * 32 + lane;
      const bool there = j <= pos_most && key_row(j) != nullptr;
#pragma unroll
      for (int x = 0; x < QS; ++x) {
        if (sq0 + x >= nq) break;
        const int pos = q_pos[sq0 + x];
        float v = s[x] * a.scale;
        if (a.softcap > 0.f) v = a.softcap * tanhf(v / a.softcap);
        v -= q_slope[sq0 + x] * (float)(pos - j);
        ps[(sq0 + x) * KT + sb * 32 + lane] = there && j <= pos && (j >= q_lo[sq0 + x] || j < a.keep_first) ? v : -INFINITY;
      }
    }
    __syncthreads();                                        // the scores are there, the keys are done with
    mine = my_row(step + 1);
    fetch(mine, ks, DK, 0);
    // all of the warp's queries and blocks at once, so that their reductions overlap; only the maxima hang on one another
    float sc[QW][KB], top[QW][KB], w[QW][KB], alpha[QW][KB];
#pragma unroll
    for (int i = 0; i < QW; ++i)
#pragma unroll
      for (int b = 0; b < KB; ++b) top[i][b] = sc[i][b] = warp + i * NW < nq ? ps[(warp + i * NW) * KT + b * 32 + lane] : -INFINITY;
    if (a.sig_bias) {
#pragma unroll
      for (int i = 0; i < QW; ++i) {
        const float bias = warp + i * NW < nq ? a.sig_bias[head0 + (warp + i * NW) % heads] : 0.f;
#pragma unroll
        for (int b = 0; b < KB; ++b) {
          alpha[i][b] = 1.f;
          w[i][b] = 1.f / (1.f + expf(-(sc[i][b] + bias)));
          top[i][b] = 0.f;
        }
      }
    } else {
#pragma unroll
      for (int o = 16; o > 0; o >>= 1)
#pragma unroll
        for (int i = 0; i < QW; ++i)
#pragma unroll
          for (int b = 0; b < KB; ++b) top[i][b] = fmaxf(top[i][b], __shfl_xor_sync(0xffffffffu, top[i][b], o));
#pragma unroll
      for (int i = 0; i < QW; ++i)
#pragma unroll
        for (int b = 0; b < KB; ++b) {
          top[i][b] = fmaxf(m[i], top[i][b]);               // -inf: nothing seen so far
          alpha[i][b] = top[i][b] == -INFINITY ? 1.f : m[i] == -INFINITY ? 0.f : expf(m[i] - top[i][b]);
          w[i][b] = sc[i][b] == -INFINITY || top[i][b] == -INFINITY ? 0.f : expf(sc[i][b] - top[i][b]);
          m[i] = top[i][b];
        }
      float sum[QW][KB];
#pragma unroll
      for (int i = 0; i < QW; ++i)
#pragma unroll
        for (int b = 0; b < KB; ++b) sum[i][b] = w[i][b];
#pragma unroll
      for (int o = 16; o > 0; o >>= 1)
#pragma unroll
        for (int i = 0; i < QW; ++i)
#pragma unroll
          for (int b = 0; b < KB; ++b) sum[i][b] += __shfl_xor_sync(0xffffffffu, sum[i][b], o);
#pragma unroll
      for (int i = 0; i < QW; ++i)
#pragma unroll
        for (int b = 0; b < KB; ++b) l[i] = l[i] * alpha[i][b] + sum[i][b];
    }
#pragma unroll
    for (int i = 0; i < QW; ++i) {
      const int x = warp + i * NW;
      if (x < nq) {
#pragma unroll
        for (int b = 0; b < KB; ++b) {
          const int j = j0 + b * 32 + lane;
          const float unseen = j > q_pos[x] || (j < q_lo[x] && j >= a.keep_first) ? -1.f : 0.f;
          ps[x * KT + b * 32 + lane] = sc[i][b] == -INFINITY || top[i][b] == -INFINITY ? unseen : w[i][b];
          if (lane == 0) as[b * Q + x] = alpha[i][b];
        }
      }
    }
    af_wait<1>();                                           // the values are in
    __syncthreads();
    if (vd < D && vq0 < nq) {
#pragma unroll 1
      for (int b = 0; b < KB; ++b) {
        if (j0 + b * 32 > pos_most) break;
        // are all these keys seen by all queries of a whole tile?  Otherwise a weight below 0 leaves its value out.
        const int live = min(32, pos_most + 1 - (j0 + b * 32));
        const bool all = j0 + b * 32 + 31 <= pos_least && j0 + b * 32 >= lo_most && nq == a.rows_tile * a.heads_tile;
#pragma unroll
        for (int x = 0; x < QV; ++x)
          if (vq0 + x < nq) {
            const float alpha = as[b * Q + vq0 + x];
#pragma unroll
            for (int i = 0; i < DI; ++i) acc[i][x] *= alpha;
          }
#pragma unroll(QV > 8 ? 1 : 2)
        for (int r = 0; r < live; r += 4) {
          const float* v = vs + (size_t)(b * 32 + r) * D + vd;
          float vv[DI][4];
#pragma unroll
          for (int i = 0; i < DI; ++i)
#pragma unroll
            for (int e = 0; e < 4; ++e) vv[i][e] = DI == 1 || vd + i * kAfThreads < D ? v[e * D + i * kAfThreads] : 0.f;
          const float* p = ps + (size_t)vq0 * KT + b * 32 + r;
          if (all) {
#pragma unroll
            for (int x = 0; x < QV; ++x) {
              float pp[4];
              load4(p + x * KT, pp);
#pragma unroll
              for (int e = 0; e < 4; ++e)
#pragma unroll
                for (int i = 0; i < DI; ++i) acc[i][x] = fmaf(pp[e], vv[i][e], acc[i][x]);
            }
          } else {
#pragma unroll
            for (int x = 0; x < QV; ++x) {
              if (vq0 + x < nq) {
                float pp[4];
                load4(p + x * KT, pp);
#pragma unroll
                for (int e = 0; e < 4; ++e)
#pragma unroll
                  for (int i = 0; i < DI; ++i) acc[i][x] = pp[e] < 0.f ? acc[i][x] : fmaf(pp[e], vv[i][e], acc[i][x]);
              }
            }
          }
        }
      }
    }
    __syncthreads();                                        // the values and weights are done with
    fetch(mine, vs, D, (size_t)a.Hkv * head_stride);
  }
  af_wait<0>();
  // 1 / l of every query, times its gate, by the warp that kept it
#pragma unroll
  for (int i = 0; i < QW; ++i) {
    const int x = warp + i * NW;
    if (x < nq && lane == 0) {
      float inv_l = a.sig_bias ? 1.f : (l[i] > 0.f ? 1.f / l[i] : 0.f);
      if (a.gate) inv_l *= 1.f / (1.f + expf(-a.gate[(size_t)(row0 + x / heads) * a.gate_ld + head0 + x % heads]));
      as[x] = inv_l;
    }
  }
  __syncthreads();
  if (vd < D) {
#pragma unroll
    for (int x = 0; x < QV; ++x) {
      const int q = vq0 + x;
      if (q < nq) {
        float* o = a.out + (size_t)(row0 + q / heads) * a.Hq * D + (size_t)(head0 + q % heads) * D;
#pragma unroll
        for (int i = 0; i < DI; ++i)
          if (vd + i * kAfThreads < D) o[vd + i * kAfThreads] = acc[i][x] * as[q];
      }
    }
  }
}

template <int Q, int KB, int DP>
__global__ void __launch_bounds__(kAfThreads)
paged_attention_f32_kernel(const AfArgs args) {
  extern __shared__ __align__(16) float af_smem[];
  __shared__ int q_pos[Q], q_lo[Q];
  __shared__ float q_slope[Q];
  AfArgs a = args;
  const int lane = threadIdx.x & 31;
  chain_wait(a.qkv, a.pages, a.gate, a.block_table, a.positions, a.row_seg, a.seg_row0);

  // which rows: the tile-th run of rows_tile rows of a segment
  AfTile t;
  if (a.rows_tile == 1) {
    t.row0 = blockIdx.x, t.rows = 1;
  } else {
    int left = blockIdx.x;
    t.rows = 0;
    for (int s0 = 0; s0 < a.S; s0 += 32) {
      const int s = s0 + lane;
      const int begin = s < a.S ? a.seg_row0[s] : 0, own_rows = s < a.S ? a.seg_row0[s + 1] - begin : 0;
      const int own = (own_rows + a.rows_tile - 1) / a.rows_tile;
      int upto = own;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int v = __shfl_up_sync(0xffffffffu, upto, o);
        if (lane >= o) upto += v;
      }
      const unsigned past = __ballot_sync(0xffffffffu, upto > left);
      if (past) {
        const int at = __ffs(past) - 1;
        left = (left - __shfl_sync(0xffffffffu, upto - own, at)) * a.rows_tile;
        t.row0 = __shfl_sync(0xffffffffu, begin, at) + left;
        t.rows = min(a.rows_tile, __shfl_sync(0xffffffffu, own_rows, at) - left);
        break;
      }
      left -= __shfl_sync(0xffffffffu, upto, 31);
    }
    if (t.rows == 0) return;                                // the grid is an upper bound
  }
  const int group = a.Hq / a.Hkv;
  t.kvh = blockIdx.y / a.head_tiles;
  t.head0 = t.kvh * group + (blockIdx.y % a.head_tiles) * a.heads_tile;
  t.heads = min(a.heads_tile, (t.kvh + 1) * group - t.head0);
  t.bt = a.block_table + (size_t)a.row_seg[t.row0] * a.bt_width;
  static_assert(Q <= 32, "a lane a row");
  const int p = a.positions[t.row0 + (lane < t.rows ? lane : 0)];
  t.pos_most = __reduce_max_sync(0xffffffffu, p);
  t.pos_least = __reduce_min_sync(0xffffffffu, p);
  // a tile whose keys are one block has it fetched and scored by all warps
  if (KB > 1 && t.pos_most < 32) af_tile<Q, 1, DP>(a, t, af_smem, q_pos, q_lo, q_slope);
  else af_tile<Q, KB, DP>(a, t, af_smem, q_pos, q_lo, q_slope);
}

template <int Q, int KB, int DP>
int af_launch(AfArgs a, int row_tiles, cudaStream_t stream) {
  const size_t smem = af_floats<Q, KB>(a.D) * sizeof(float);
  static const cudaError_t e = cudaFuncSetAttribute(paged_attention_f32_kernel<Q, KB, DP>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                                    (int)(af_floats<Q, KB>(DP) * sizeof(float)));
  NF_REQUIRE(e == cudaSuccess, "attention: cannot have %zu bytes of shared memory: %s", smem, cudaGetErrorString(e));
  launch_chained(paged_attention_f32_kernel<Q, KB, DP>, dim3(row_tiles, a.Hkv * a.head_tiles), dim3(kAfThreads), smem, stream, a);
  return check_launch("paged_attention_f32");
}

// CTAs of this form that a SM holds beside one another: by their shared memory (228 KB, 1 KB of it taken by each CTA), and
// by their registers six
template <int Q, int KB>
int af_resident(int D) {
  const int fit = (int)(228 * 1024 / (af_floats<Q, KB>(D) * sizeof(float) + 1024));
  return fit < 6 ? fit : 6;
}

template <int Q, int KB>
int af_heads(const AfArgs& a, int row_tiles, cudaStream_t stream) {
  if (a.D <= 32) return af_launch<Q, KB, 32>(a, row_tiles, stream);
  if (a.D <= 64) return af_launch<Q, KB, 64>(a, row_tiles, stream);
  if (a.D <= 128) return af_launch<Q, KB, 128>(a, row_tiles, stream);
  return af_launch<Q, (KB < 2 ? KB : 2), 256>(a, row_tiles, stream);       // four blocks of such rows do not fit
}

// The form of most blocks at a time (up to MOST) whose CTAs all lie beside one another; figures at the top.  (Four queries
// of more than 64 dimensions gain nothing from four blocks: 4 rows of 28 heads over 1,024 keys 87 us with two, 88 with four.)
template <int Q, int MOST>
int af_blocks(const AfArgs& a, int row_tiles, cudaStream_t stream) {
  const long long ctas = (long long)row_tiles * a.Hkv * a.head_tiles;
  if (MOST >= 4 && ctas <= 148ll * af_resident<Q, 4>(a.D)) return af_heads<Q, (MOST >= 4 ? 4 : 1)>(a, row_tiles, stream);
  if (ctas <= 148ll * af_resident<Q, 2>(a.D)) return af_heads<Q, 2>(a, row_tiles, stream);
  return af_heads<Q, 1>(a, row_tiles, stream);
}

}  // namespace
}  // namespace nf

using namespace nf;

// Head sizes up to 256 that are multiples of 4, pages on 16 bytes.  `seg_row0` int32 [S + 1]: the segments' first rows;
// `max_rows`: the most rows of a segment in this step (1: every row is its own segment's only one).
extern "C" int nf_paged_attention_f32(const float* qkv, int q_row_stride, const float* pages, const int* block_table, int bt_width,
                                      const int* positions, const int* row_seg, const int* seg_row0, int S, int max_rows,
                                      float* out, int T, int Hq, int Hkv, int D, int page_size, int num_pages, int window,
                                      float scale, const float* slopes, int keep_first, const float* gate, int gate_ld,
                                      const float* sig_bias, float softcap, cudaStream_t stream) {
  if (T == 0) return 0;
  NF_REQUIRE(T > 0 && Hq > 0 && Hkv > 0 && Hq % Hkv == 0 && S > 0, "attention: bad sizes T=%d S=%d Hq=%d Hkv=%d", T, S, Hq, Hkv);
  NF_REQUIRE(D >= 4 && D <= 256 && D % 4 == 0 && (uintptr_t)pages % 16 == 0, "attention: head_dim %d or pages not in 16-byte pieces", D);
  AfArgs a{qkv, pages, block_table, positions, row_seg, seg_row0, out, slopes, gate, sig_bias, q_row_stride, bt_width, T, S, Hq,
           Hkv, D, page_size, num_pages, window, window > 0 ? keep_first : 0, gate_ld, 0, 0, 0, scale, softcap};
  const int group = Hq / Hkv;
  const int q = max_rows > 1 ? (group > 8 ? 16 : 8) : group > 2 ? 4 : group;
  a.heads_tile = group < q ? group : q;
  a.rows_tile = max_rows > 1 ? q / a.heads_tile : 1;
  a.head_tiles = (group + a.heads_tile - 1) / a.heads_tile;
  NF_REQUIRE((long long)Hkv * a.head_tiles <= 65535, "attention: too many heads (%d)", Hq);
  const long long tiles = a.rows_tile == 1 ? T : (long long)T / a.rows_tile + S < T ? T / a.rows_tile + S : T;
  if (q == 16) return af_blocks<16, 2>(a, (int)tiles, stream);
  if (q == 8) return af_blocks<8, 2>(a, (int)tiles, stream);
  if (q == 4) return D <= 64 ? af_blocks<4, 4>(a, (int)tiles, stream) : af_blocks<4, 2>(a, (int)tiles, stream);
  if (q == 2) return af_blocks<2, 4>(a, (int)tiles, stream);
  return af_blocks<1, 4>(a, (int)tiles, stream);
}
