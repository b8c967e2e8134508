// The recurrences  S_t = a_t S_{t-1} + w_t k_t v_t^T,  o_t = S_t^T q_t  of prompt portions on tensor cores (bfloat16
// engines): the selective scan of ssm.cu (k = B, q = C, v = x, w = dt) and the linear attention of
// linear_attention.cu (w = 1, a constant decay a head); and the gated delta rule of delta_rule.cu (further down).
// S is V x D per head, float32.
//
// Walking the rows one by one is bound by the chain from row to row (a prompt of 2,048 tokens, 64 heads of
// 128 x 64: 755 us, about 1 % of the arithmetic's own time).  Over a chunk of Q rows the recurrence is three products:
//
//   o_t  = A_t S_0^T q_t + sum_{s <= t} (D(s, t) w_s q_t.k_s) v_s      A_t = a_1 ... a_t, D(s, t) = a_{s+1} ... a_t
//   S_Q  = A_Q S_0 + sum_s D(s, Q) w_s k_s v_s^T
//
// so a step runs as (1) every chunk's own contribution to the state, all chunks and heads at once, (2) the chain over
// the chunks' states, elementwise, which leaves in a chunk's place the state it starts from, (3) the outputs of all
// chunks and heads at once.  Chunks are counted from a segment's first row of the step.  Decays are products, never
// quotients or differences of logarithms, so a decay near zero does no harm.
//
// A row's result holds what the rows up to it hold and nothing of the later ones, whatever their numbers are: a zero weight
// is no protection from an infinity or a NaN (0 * inf), so on the diagonal the scores of later keys are left out by a
// choice, and a product there that came out other than finite is done again without the values that are not.
//
// Everything beyond the activations stays float32 in what it carries: a float32 operand goes to the bfloat16 tensor
// cores as three bfloat16 parts (8 + 8 + 8 bits: the number itself), a bfloat16 one as it is, and the partial
// products whose weight is at least 2^-16 of the leading one are all taken (three where one operand is bfloat16, six
// where both are float32) with float32 sums.
//
// One prompt of 2,048 tokens, row by row and now: scan of 64 heads of 128 x 64 755 and 135 us (under a profiler, from a cold
// cache, the outputs 95, the chunks' states 47, the chain over 16 chunks, which moves 67 MB, 15), 32 heads of 64 x 64 394 and 57;
// linear attention of 16 heads of 128 x 128 with float32 q, k and v 499 and 150 (outputs 95, states 41, chain 22), 64 x 128 with
// bfloat16 values 347 and 74; the delta rule of 16 heads of 128 x 128 431 and 172.  Chunks of 128 rows halve the states' traffic where the operands are bfloat16; with three parts of each
// operand in shared memory 64 rows fit.
#define NF_CHAIN_CLASS 2
#include "common.cuh"

namespace nf {
namespace {

constexpr int kCrThreads = 256;
constexpr int kCrPad = 8;               // elements of padding a shared-memory row: ldmatrix then meets no bank conflict

enum CrMode : int { kCrScan = 0, kCrDecay = 1, kCrDelta = 2 };

// Which chunks a launch serves: those of the segments of at least min_rows rows, counted over all of them, from chunk
// `first` on, and of these segments those from number `first_run` on.  Where they lie is worked out on the device from the
// step's own index of rows: lists of chunks and runs made on the host cost a step of few rows, which waits for its host,
// more than the recurrence itself (one scan of 256 rows: 24 us to build and send them).
struct CrChunks {
  const int* seg_row0;
  int S, min_rows, first, n, first_run;
};
struct CrPlace {
  int seg, row0, rows, chunk;           // a segment, its first row, its rows, the number of its first chunk
};
// The segment of chunk `c`, or (RUN) the segment of number `c`; a warp's lanes look at 32 segments at a time.  The index is
// a step's input, complete before the step's kernels began.
template <int Q, bool RUN>
__device__ __forceinline__ CrPlace cr_find(const CrChunks& at, int c) {
  const int lane = threadIdx.x & 31;
  int chunks = 0, runs = 0;
  for (int s0 = 0; s0 < at.S; s0 += 32) {
    const int s = s0 + lane, row0 = s < at.S ? at.seg_row0[s] : 0, rows = s < at.S ? at.seg_row0[s + 1] - row0 : 0;
    const bool mine = rows >= at.min_rows;
    const int k = mine ? (rows + Q - 1) / Q : 0;
    int incl = k;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int up = __shfl_up_sync(0xffffffffu, incl, o);
      if (lane >= o) incl += up;
    }
    const unsigned b = __ballot_sync(0xffffffffu, mine);
    const int number = runs + __popc(b & ((1u << lane) - 1u)), first = chunks + incl - k;
    const unsigned hit = __ballot_sync(0xffffffffu, mine && (RUN ? number == c : c >= first && c < first + k));
    if (hit) {
      const int src = __ffs(hit) - 1;
      return {s0 + src, __shfl_sync(0xffffffffu, row0, src), __shfl_sync(0xffffffffu, rows, src), __shfl_sync(0xffffffffu, first, src)};
    }
    chunks += __shfl_sync(0xffffffffu, incl, 31);
    runs += __popc(b);
  }
  return {0, 0, 0, 0};                  // (no such chunk: no rows)
}
// First row and rows of chunk `c` of the launch.
template <int Q>
__device__ __forceinline__ int2 cr_rows(const CrChunks& at, int c) {
  const CrPlace p = cr_find<Q, false>(at, at.first + c);
  const int off = (at.first + c - p.chunk) * Q;
  return make_int2(p.row0 + off, max(0, min(Q, p.rows - off)));
}
// Of a segment's chunks those in the launch: x the first one's number in the launch, y how many, z its number in the segment.
template <int Q>
__device__ __forceinline__ int3 cr_run(const CrChunks& at, const CrPlace& p) {
  const int lo = max(p.chunk, at.first), hi = min(p.chunk + (p.rows + Q - 1) / Q, at.first + at.n);
  return make_int3(lo - at.first, max(0, hi - lo), lo - p.chunk);
}

struct CrArgs {
  const __nv_bfloat16 *q, *k, *v;       // rows of `ld` elements, columns from q0, k0, v0 on (q and k: a head group's D)
  int ld, q0, k0, v0;
  const float* prepared;                // float32 q and k [T, 2, H, D] instead
  int v_silu;
  int H, heads_per_group, V;
  const __nv_bfloat16* dt;              // scan: raw step sizes
  int ld_dt, dt0;
  const float *dt_bias, *A_log, *skip;
  const float* decay;                   // a decay a head
  const float* values;                  // delta rule: float32 values [T, H * V] (u), and [T, H, 4] of (decay, factor on
  const float* gates;                   // the row's key, factor on its output, -)
  CrChunks at;
  const int* seg_slot;
  float* state;
  long slot_stride;
  float* chunk_state;                   // [n][H][V][D]
  float* chunk_decay;                   // [n][H]
  float* out;                           // [T][H * V]
};

__device__ __forceinline__ unsigned cr_smem(const void* p) { return (unsigned)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void cr_ldm4(unsigned addr, unsigned (&r)[4]) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr) : "memory");
}
__device__ __forceinline__ void cr_ldm4t(unsigned addr, unsigned (&r)[4]) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr) : "memory");
}
__device__ __forceinline__ void cr_mma(float (&c)[4], const unsigned (&a)[4], unsigned b0, unsigned b1) {
  asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
               : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3]) : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
// The tensor cores cut a sum off where float32 arithmetic rounds it, always towards zero: over the 48 products that a sum
// of 128 terms in parts takes this adds up (linear attention of 64 rows, D = 128: 9.7e-7 of the results, row by row in
// float32 1.6e-7).  So the products of one step of 16 terms start from zero, the smallest parts first, and their sum is
// added to the running one in float32: 1.5e-7, and over 2,048 rows 3.0e-7 against 8.0e-7 row by row.  It
// costs a scan 3 %, 128 x 128 with six products a step 16 %.
template <int N>
__device__ __forceinline__ void cr_zero(float (&t)[N][4]) {
#pragma unroll
  for (int n = 0; n < N; ++n)
#pragma unroll
    for (int e = 0; e < 4; ++e) t[n][e] = 0.f;
}
__device__ __forceinline__ void cr_add(float (&c)[4], const float (&t)[4]) {
#pragma unroll
  for (int e = 0; e < 4; ++e) c[e] += t[e];
}
__device__ __forceinline__ bool cr_finite(const float (&t)[4]) {
  return fabsf(t[0]) < INFINITY && fabsf(t[1]) < INFINITY && fabsf(t[2]) < INFINITY && fabsf(t[3]) < INFINITY;
}
// A packed pair with zeros for what is not finite.
__device__ __forceinline__ unsigned cr_finite_only(unsigned x) {
  if ((x & 0x7f800000u) == 0x7f800000u) x &= 0x0000ffffu;
  if ((x & 0x00007f80u) == 0x00007f80u) x &= 0xffff0000u;
  return x;
}
// Two neighbouring numbers as PARTS packed pairs of bfloat16 that add up to them.  What has no remainder (an infinity,
// a NaN) stands in the first part alone.
template <int PARTS>
__device__ __forceinline__ void cr_split(float x, float y, unsigned (&p)[PARTS]) {
#pragma unroll
  for (int i = 0; i < PARTS; ++i) {
    const __nv_bfloat162 h = __floats2bfloat162_rn(x, y);
    p[i] = *reinterpret_cast<const unsigned*>(&h);
    if (i + 1 < PARTS) {
      const float hx = __low2float(h), hy = __high2float(h);
      x = isinf(hx) || isnan(hx) ? 0.f : x - hx;
      y = isinf(hy) || isnan(hy) ? 0.f : y - hy;
    }
  }
}
// Four consecutive numbers to the same place of PARTS planes.
template <int PARTS>
__device__ __forceinline__ void cr_store_parts(__nv_bfloat16* dst, size_t plane, const float (&x)[4]) {
  unsigned lo[PARTS], hi[PARTS];
  cr_split<PARTS>(x[0], x[1], lo);
  cr_split<PARTS>(x[2], x[3], hi);
#pragma unroll
  for (int i = 0; i < PARTS; ++i) *reinterpret_cast<uint2*>(dst + i * plane) = make_uint2(lo[i], hi[i]);
}

// The chunk's decays and weights, one thread a row: 1 and 0 beyond its rows, so that those count nothing.
template <int MODE>
__device__ __forceinline__ void cr_row_gates(const CrArgs& a, int head, int row, bool live, float& decay, float& weight) {
  decay = 1.f;
  weight = 0.f;
  if (!live) return;
  if (MODE == kCrScan) {
    const float v = to_float(a.dt[(size_t)row * a.ld_dt + a.dt0 + head]) + a.dt_bias[head];
    weight = v > 20.f ? v : log1pf(expf(v));
    decay = expf(-expf(a.A_log[head]) * weight);
  } else if (MODE == kCrDecay) {
    decay = a.decay[head];
    weight = 1.f;
  } else {
    const float2 g = *reinterpret_cast<const float2*>(a.gates + ((size_t)row * a.H + head) * 4);
    decay = g.x;
    weight = g.y;
  }
}

// What a chunk's CTA reads goes through registers in two halves: `ask` issues every load, `put` brings the numbers to
// shared memory (in parts, where they are float32).  Between the two lies other work - gates, decay tables, the products
// with the rows or the state before - so that a CTA, of which only two fit a SM, does not stand still for each of its reads
// (with loads and stores in one loop the scan of 2,048 rows above took 164 us, linear attention 213, the delta rule 197).
//
// ROWS rows of the keys (or queries) for planes [PARTS][.][D + pad]; zeros from `live` rows on.
template <int D, int PARTS, int ROWS>
struct CrQkRows {
  static constexpr int W = PARTS == 1 ? 8 : 4, N = ROWS * (D / W) / kCrThreads;
  static_assert(ROWS * (D / W) % kCrThreads == 0, "whole rounds of loads");
  uint4 x[N];
  __device__ __forceinline__ void ask(const CrArgs& a, bool keys, int head, int row0, int live) {
#pragma unroll
    for (int i = 0; i < N; ++i) {
      const int at = threadIdx.x + i * kCrThreads, r = at / (D / W), c = (at % (D / W)) * W;
      x[i] = make_uint4(0, 0, 0, 0);
      if (r < live) {
        if (PARTS == 1)
          x[i] = *reinterpret_cast<const uint4*>((keys ? a.k + a.k0 : a.q + a.q0) + (size_t)(head / a.heads_per_group) * D + (size_t)(row0 + r) * a.ld + c);
        else
          x[i] = *reinterpret_cast<const uint4*>(a.prepared + (size_t)(keys ? a.H + head : head) * D + (size_t)(row0 + r) * 2 * a.H * D + c);
      }
    }
  }
  __device__ __forceinline__ void put(__nv_bfloat16* dst, size_t plane) const {
#pragma unroll
    for (int i = 0; i < N; ++i) {
      const int at = threadIdx.x + i * kCrThreads, r = at / (D / W), c = (at % (D / W)) * W;
      if (PARTS == 1) {
        *reinterpret_cast<uint4*>(dst + r * (D + kCrPad) + c) = x[i];
      } else {
        const float f[4] = {__uint_as_float(x[i].x), __uint_as_float(x[i].y), __uint_as_float(x[i].z), __uint_as_float(x[i].w)};
        cr_store_parts<PARTS>(dst + r * (D + kCrPad) + c, plane, f);
      }
    }
  }
};
__device__ __forceinline__ float cr_value(float x, int silu) { return silu ? x / (1.f + expf(-x)) : x; }
// ROWS rows of V columns of a head's values from column `col` on, for planes [PARTS][.][V + pad]: bfloat16 as they are
// (PARTS 1), through the activation and times a row's `scale` (null: 1), or (FLOATS) the float32 numbers of `values`.
template <int V, int PARTS, int ROWS, bool FLOATS>
struct CrValueRows {
  static constexpr int W = PARTS == 1 ? 8 : 4, N = ROWS * (V / W) / kCrThreads;
  static_assert(ROWS * (V / W) % kCrThreads == 0 && !(FLOATS && PARTS == 1), "whole rounds of loads");
  uint4 x[N];
  __device__ __forceinline__ void ask(const CrArgs& a, int head, int col, int row0, int live) {
#pragma unroll
    for (int i = 0; i < N; ++i) {
      const int at = threadIdx.x + i * kCrThreads, r = at / (V / W), c = (at % (V / W)) * W;
      x[i] = make_uint4(0, 0, 0, 0);
      if (r < live) {
        if (FLOATS) {
          x[i] = *reinterpret_cast<const uint4*>(a.values + (size_t)(row0 + r) * a.H * a.V + (size_t)head * a.V + col + c);
        } else {
          const __nv_bfloat16* src = a.v + a.v0 + (size_t)head * a.V + col + (size_t)(row0 + r) * a.ld + c;
          if (PARTS == 1) {
            x[i] = *reinterpret_cast<const uint4*>(src);
          } else {
            const uint2 half = *reinterpret_cast<const uint2*>(src);
            x[i].x = half.x, x[i].y = half.y;
          }
        }
      }
    }
  }
  __device__ __forceinline__ void put(__nv_bfloat16* dst, size_t plane, int silu, const float* scale) const {
#pragma unroll
    for (int i = 0; i < N; ++i) {
      const int at = threadIdx.x + i * kCrThreads, r = at / (V / W), c = (at % (V / W)) * W;
      if (PARTS == 1) {
        *reinterpret_cast<uint4*>(dst + r * (V + kCrPad) + c) = x[i];
        continue;
      }
      float f[4] = {__uint_as_float(x[i].x), __uint_as_float(x[i].y), __uint_as_float(x[i].z), __uint_as_float(x[i].w)};
      if (!FLOATS) {
        const uint2 half = make_uint2(x[i].x, x[i].y);
        load4(reinterpret_cast<const __nv_bfloat16*>(&half), f);
#pragma unroll
        for (int e = 0; e < 4; ++e) f[e] = cr_value(f[e], silu);
        if (scale) {
          const float by = scale[r];
#pragma unroll
          for (int e = 0; e < 4; ++e) f[e] *= by;
        }
      }
      cr_store_parts<PARTS>(dst + r * (V + kCrPad) + c, plane, f);
    }
  }
};
// Row t's decays inside its sixteen, from the chunk's in `decay`: the product up to it, after it, and to every later row
// (diag[t / 16][t % 16][u]; 0 before it).
template <int N>
__device__ __forceinline__ void cr_decay_table(const float* decay, int t, float* upto, float* after, float (&diag)[N][16][17]) {
  const int b = t & ~15;
  float run = 1.f;
  for (int s = b; s <= t; ++s) run *= decay[s];
  upto[t] = run;
  run = 1.f;
  for (int u = 0; u < 16; ++u) {
    if (b + u > t) run *= decay[b + u];
    diag[t >> 4][t & 15][u] = b + u < t ? 0.f : run;
  }
  after[t] = run;
}

// ---- (1) a chunk's contribution to the state: [V, D] = sum_s (w_s D(s, end) v_s) k_s^T -------------------------------
// 8 warps: a warp owns 32 value rows and D V / 256 state columns.
template <int D, int V, int Q, int QKP, int MODE>
__global__ void __launch_bounds__(kCrThreads, 2)
chunk_state_kernel(const CrArgs args) {
  constexpr int WM = V / 32, WN = 8 / WM, NT = D / WN / 8;     // warps along V and D, column tiles a warp
  constexpr int KS = D + kCrPad, VS = V + kCrPad;
  static_assert(V % 32 == 0 && 8 % WM == 0 && D % (WN * 16) == 0 && Q % 32 == 0 && Q <= kCrThreads, "chunk shape");
  extern __shared__ __align__(16) unsigned char cr_raw[];
  __nv_bfloat16* Ks = reinterpret_cast<__nv_bfloat16*>(cr_raw);              // [QKP][Q][KS]
  __nv_bfloat16* Vs = Ks + (size_t)QKP * Q * KS;                             // [3][Q][VS]
  __shared__ float s_decay[Q], s_scale[Q];
  const int chunk = blockIdx.x, head = blockIdx.y;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  CrArgs a = args;
  const int2 place = cr_rows<Q>(a.at, chunk);
  const int row0 = place.x, live = place.y;
  chain_wait(a.q, a.k, a.v, a.dt, a.prepared);
  CrQkRows<D, QKP, Q> keys;
  CrValueRows<V, 3, Q, false> values;
  keys.ask(a, true, head, row0, live);
  values.ask(a, head, 0, row0, live);
  float weight = 0.f;
  if (threadIdx.x < Q) {
    float decay;
    cr_row_gates<MODE>(a, head, row0 + threadIdx.x, (int)threadIdx.x < live, decay, weight);
    s_decay[threadIdx.x] = decay;
  }
  __syncthreads();
  if (threadIdx.x < Q) {                 // w_s D(s, end): the rows after s in its 16, then whole sixteens
    float run = 1.f;
    const int end = (threadIdx.x & ~15) + 16;
    for (int s = threadIdx.x + 1; s < end; ++s) run *= s_decay[s];
    s_scale[threadIdx.x] = run;          // decays after s to the end of its sixteen
  }
  __syncthreads();
  if (threadIdx.x < Q) {
    float run = s_scale[threadIdx.x];
    for (int b = (threadIdx.x >> 4) + 1; b < Q / 16; ++b) run *= s_scale[16 * b] * s_decay[16 * b];
    if (threadIdx.x == 0) a.chunk_decay[(size_t)chunk * a.H + head] = run * s_decay[0];
    weight *= run;
  }
  __syncthreads();
  if (threadIdx.x < Q) s_scale[threadIdx.x] = weight;
  keys.put(Ks, (size_t)Q * KS);
  __syncthreads();
  values.put(Vs, (size_t)Q * VS, a.v_silu, s_scale);
  __syncthreads();
  const int m0 = (warp % WM) * 32, n0 = (warp / WM) * (D / WN);
  float acc[2][NT][4];
#pragma unroll
  for (int m = 0; m < 2; ++m)
#pragma unroll
    for (int n = 0; n < NT; ++n)
#pragma unroll
      for (int e = 0; e < 4; ++e) acc[m][n][e] = 0.f;
  const int mat = lane >> 3, r8 = lane & 7;
  const unsigned va = cr_smem(Vs + ((mat >> 1) * 8 + r8) * VS + m0 + (mat & 1) * 8);
  const unsigned ka = cr_smem(Ks + ((mat & 1) * 8 + r8) * KS + n0 + (mat >> 1) * 8);
#pragma unroll 1
  for (int s0 = 0; s0 < Q; s0 += 16) {
    if (s0 >= live) break;
    unsigned A[3][2][4];
#pragma unroll
    for (int i = 0; i < 3; ++i)
#pragma unroll
      for (int m = 0; m < 2; ++m) cr_ldm4t(va + ((i * Q + s0) * VS + m * 16) * 2, A[i][m]);
#pragma unroll
    for (int n = 0; n < NT; n += 2) {
      float t[4][4];
      cr_zero(t);
#pragma unroll
      for (int j = QKP - 1; j >= 0; --j) {
        unsigned B[4];
        cr_ldm4t(ka + ((j * Q + s0) * KS + n * 8) * 2, B);
#pragma unroll
        for (int i = 2 - j; i >= 0; --i)
#pragma unroll
          for (int m = 0; m < 2; ++m) {
            cr_mma(t[2 * m], A[i][m], B[0], B[1]);
            cr_mma(t[2 * m + 1], A[i][m], B[2], B[3]);
          }
      }
#pragma unroll
      for (int m = 0; m < 2; ++m) {
        cr_add(acc[m][n], t[2 * m]);
        cr_add(acc[m][n + 1], t[2 * m + 1]);
      }
    }
  }
  float* dst = a.chunk_state + ((size_t)chunk * a.H + head) * V * D;
#pragma unroll
  for (int m = 0; m < 2; ++m)
#pragma unroll
    for (int n = 0; n < NT; ++n) {
      float* p = dst + (size_t)(m0 + m * 16 + (lane >> 2)) * D + n0 + n * 8 + (lane & 3) * 2;
      *reinterpret_cast<float2*>(p) = make_float2(acc[m][n][0], acc[m][n][1]);
      *reinterpret_cast<float2*>(p + 8 * D) = make_float2(acc[m][n][2], acc[m][n][3]);
    }
}

// ---- (2) the chain over a segment's chunks --------------------------------------------------------------------------
// A thread carries four of a head's V D state entries through the segment's chunks; loads run four chunks ahead.
template <int Q>
__global__ void __launch_bounds__(kCrThreads)
chunk_chain_kernel(const CrArgs args, int entries) {
  constexpr int AHEAD = 4;
  const int run = blockIdx.x, head = blockIdx.y, e = (blockIdx.z * kCrThreads + threadIdx.x) * 4;
  CrArgs a = args;
  const CrPlace place = cr_find<Q, true>(a.at, a.at.first_run + run);
  const int3 own = cr_run<Q>(a.at, place);
  const int seg = place.seg, first = own.x, n = own.y;
  chain_wait(a.chunk_state, a.chunk_decay, a.state);
  if (e >= entries) return;
  float* slot = a.state + (size_t)a.seg_slot[seg] * a.slot_stride + (size_t)head * entries + e;
  float* mine = a.chunk_state + ((size_t)first * a.H + head) * entries + e;
  const float* decay = a.chunk_decay + (size_t)first * a.H + head;
  const size_t step = (size_t)a.H * entries;
  float4 s = *reinterpret_cast<const float4*>(slot);
  float4 next[AHEAD];
  float d[AHEAD];
#pragma unroll
  for (int i = 0; i < AHEAD; ++i)
    if (i < n) {
      next[i] = *reinterpret_cast<const float4*>(mine + i * step);
      d[i] = decay[(size_t)i * a.H];
    }
  for (int c0 = 0; c0 < n; c0 += AHEAD)
#pragma unroll
    for (int i = 0; i < AHEAD; ++i) {
      const int c = c0 + i;
      if (c < n) {
        const float4 x = next[i];
        const float f = d[i];
        *reinterpret_cast<float4*>(mine + c * step) = s;
        if (c + AHEAD < n) {
          next[i] = *reinterpret_cast<const float4*>(mine + (c + AHEAD) * step);
          d[i] = decay[(size_t)(c + AHEAD) * a.H];
        }
        s.x = fmaf(f, s.x, x.x);
        s.y = fmaf(f, s.y, x.y);
        s.z = fmaf(f, s.z, x.z);
        s.w = fmaf(f, s.w, x.w);
      }
    }
  *reinterpret_cast<float4*>(slot) = s;
}

// ---- (3) a chunk's outputs --------------------------------------------------------------------------------------------
// A CTA has V of a head's a.V columns, a warp 16 rows and V / (8 / (Q / 16)) columns.  Shared memory holds the queries
// throughout; beside them first the state at the chunk's start, then the keys and values, SUB rows at a time.
template <int D, int V, int Q, int SUB, int QKP, int VP, int MODE>
__global__ void __launch_bounds__(kCrThreads, 2)
chunk_output_kernel(const CrArgs args) {
  constexpr int WQ = Q / 16, WV = 8 / WQ, NT = V / WV / 8;
  constexpr int KS = D + kCrPad, VS = V + kCrPad;
  static_assert(WQ * WV == 8 && NT % 2 == 0 && Q % SUB == 0 && SUB % 16 == 0, "chunk shape");
  extern __shared__ __align__(16) unsigned char cr_raw[];
  __nv_bfloat16* Qs = reinterpret_cast<__nv_bfloat16*>(cr_raw);              // [QKP][Q][KS]
  __nv_bfloat16* Ss = Qs + (size_t)QKP * Q * KS;                             // [3][V][KS]
  __nv_bfloat16* Ks = Ss;                                                    // [QKP][SUB][KS]
  __nv_bfloat16* Vs = Ks + (size_t)QKP * SUB * KS;                           // [VP][SUB][VS]
  __shared__ float s_decay[Q], s_weight[Q], s_upto[Q], s_after[Q];
  __shared__ float s_diag[WQ][16][17];                                       // [.][s][t]: D(s, t) inside a sixteen
  const int chunk = blockIdx.x, head = blockIdx.y, tile0 = blockIdx.z * V;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  CrArgs a = args;
  const int2 place = cr_rows<Q>(a.at, chunk);
  const int row0 = place.x, live = place.y;
  chain_wait(a.q, a.k, a.v, a.dt, a.prepared, a.chunk_state, a.values, a.gates);
  CrQkRows<D, QKP, Q> queries;
  constexpr int SN = V * (D / 4) / kCrThreads;
  static_assert(V * (D / 4) % kCrThreads == 0, "whole rounds of loads");
  float start[SN][4];                    // the state at the chunk's start
  queries.ask(a, false, head, row0, live);
  {
    const float* src = a.chunk_state + (((size_t)chunk * a.H + head) * a.V + tile0) * D;
#pragma unroll
    for (int i = 0; i < SN; ++i) load4(src + (size_t)(threadIdx.x + i * kCrThreads) * 4, start[i]);
  }
  if (threadIdx.x < Q)
    cr_row_gates<MODE>(a, head, row0 + threadIdx.x, (int)threadIdx.x < live, s_decay[threadIdx.x], s_weight[threadIdx.x]);
  queries.put(Qs, (size_t)Q * KS);
#pragma unroll
  for (int i = 0; i < SN; ++i) {
    const int at = threadIdx.x + i * kCrThreads;
    cr_store_parts<3>(Ss + (at / (D / 4)) * KS + (at % (D / 4)) * 4, (size_t)V * KS, start[i]);
  }
  CrQkRows<D, QKP, SUB> keys;            // the next SUB rows
  CrValueRows<V, VP, SUB, MODE == kCrDelta> values;
  keys.ask(a, true, head, row0, live);
  values.ask(a, head, tile0, row0, live);
  __syncthreads();
  if (threadIdx.x < Q) cr_decay_table(s_decay, threadIdx.x, s_upto, s_after, s_diag);
  __syncthreads();
  const int rb = warp % WQ, n0 = (warp / WQ) * (V / WV);       // this warp's sixteen and first column
  const int g = lane >> 2, t4 = lane & 3, mat = lane >> 3, r8 = lane & 7;
  const bool work = rb * 16 < live;
  float acc[NT][4];
#pragma unroll
  for (int n = 0; n < NT; ++n)
#pragma unroll
    for (int e = 0; e < 4; ++e) acc[n][e] = 0.f;
  // rows as A (and, with eight rows more first, as B of two column tiles)
  const unsigned qa = cr_smem(Qs + (rb * 16 + (mat & 1) * 8 + r8) * KS + (mat >> 1) * 8);
  if (work) {
    const unsigned sa = cr_smem(Ss + (n0 + (mat >> 1) * 8 + r8) * KS + (mat & 1) * 8);
#pragma unroll 2
    for (int k0 = 0; k0 < D; k0 += 16) {
      unsigned A[QKP][4];
#pragma unroll
      for (int i = 0; i < QKP; ++i) cr_ldm4(qa + (i * Q * KS + k0) * 2, A[i]);
#pragma unroll
      for (int n = 0; n < NT; n += 2) {
        float t[2][4];
        cr_zero(t);
#pragma unroll
        for (int j = 2; j >= 0; --j) {
          unsigned B[4];
          cr_ldm4(sa + ((j * V + n * 8) * KS + k0) * 2, B);
#pragma unroll
          for (int i = (2 - j < QKP - 1 ? 2 - j : QKP - 1); i >= 0; --i) {
            cr_mma(t[0], A[i], B[0], B[1]);
            cr_mma(t[1], A[i], B[2], B[3]);
          }
        }
        cr_add(acc[n], t[0]);
        cr_add(acc[n + 1], t[1]);
      }
    }
    float before = 1.f;                  // decays from the chunk's start to the sixteen's
    for (int b = 0; b < rb; ++b) before *= s_upto[16 * b + 15];
    const float f0 = before * s_upto[rb * 16 + g], f1 = before * s_upto[rb * 16 + g + 8];
#pragma unroll
    for (int n = 0; n < NT; ++n) {
      acc[n][0] *= f0; acc[n][1] *= f0;
      acc[n][2] *= f1; acc[n][3] *= f1;
    }
  }
  const float u0 = s_upto[rb * 16 + g], u1 = s_upto[rb * 16 + g + 8];
  const unsigned kb = cr_smem(Ks + ((mat >> 1) * 8 + r8) * KS + (mat & 1) * 8);
  const unsigned vb = cr_smem(Vs + ((mat & 1) * 8 + r8) * VS + n0 + (mat >> 1) * 8);
#pragma unroll 1
  for (int sub = 0; sub < Q; sub += SUB) {
    if (sub >= live) break;
    __syncthreads();                     // everyone is done with the state, or with the rows before
    keys.put(Ks, (size_t)SUB * KS);
    values.put(Vs, (size_t)SUB * VS, a.v_silu, nullptr);
    __syncthreads();
    if (sub + SUB < live) {
      keys.ask(a, true, head, row0 + sub + SUB, live - sub - SUB);
      values.ask(a, head, tile0, row0 + sub + SUB, live - sub - SUB);
    }
    if (!work) continue;
#pragma unroll 1
    for (int sb = 0; sb < SUB; sb += 16) {
      const int b = (sub + sb) >> 4;     // the sixteen of keys
      if (b > rb) break;
      float p[2][4];
#pragma unroll
      for (int n = 0; n < 2; ++n)
#pragma unroll
        for (int e = 0; e < 4; ++e) p[n][e] = 0.f;
#pragma unroll 2
      for (int k0 = 0; k0 < D; k0 += 16) {
        unsigned A[QKP][4];
#pragma unroll
        for (int i = 0; i < QKP; ++i) cr_ldm4(qa + (i * Q * KS + k0) * 2, A[i]);
        float t[2][4];
        cr_zero(t);
#pragma unroll
        for (int j = QKP - 1; j >= 0; --j) {
          unsigned B[4];
          cr_ldm4(kb + ((j * SUB + sb) * KS + k0) * 2, B);
#pragma unroll
          for (int i = (2 - j < QKP - 1 ? 2 - j : QKP - 1); i >= 0; --i) {
            cr_mma(t[0], A[i], B[0], B[1]);
            cr_mma(t[1], A[i], B[2], B[3]);
          }
        }
        cr_add(p[0], t[0]);
        cr_add(p[1], t[1]);
      }
      // times D(s, t) w_s
      if (b == rb) {
#pragma unroll
        for (int n = 0; n < 2; ++n)
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            const int s = n * 8 + t4 * 2 + (e & 1), t = g + (e >> 1) * 8;
            p[n][e] = s > t ? 0.f : p[n][e] * (s_diag[rb][s][t] * s_weight[b * 16 + s]);
          }
      } else {
        float between = 1.f;
        for (int x = b + 1; x < rb; ++x) between *= s_upto[16 * x + 15];
#pragma unroll
        for (int n = 0; n < 2; ++n)
#pragma unroll
          for (int e = 0; e < 2; ++e) {
            const int s = b * 16 + n * 8 + t4 * 2 + e;
            const float f = s_after[s] * between;
            const float w = s_weight[s];
            p[n][e] *= f * u0 * w;
            p[n][e + 2] *= f * u1 * w;
          }
      }
      unsigned P[3][4];
      {
        unsigned x[3];
        cr_split<3>(p[0][0], p[0][1], x);
        P[0][0] = x[0]; P[1][0] = x[1]; P[2][0] = x[2];
        cr_split<3>(p[0][2], p[0][3], x);
        P[0][1] = x[0]; P[1][1] = x[1]; P[2][1] = x[2];
        cr_split<3>(p[1][0], p[1][1], x);
        P[0][2] = x[0]; P[1][2] = x[1]; P[2][2] = x[2];
        cr_split<3>(p[1][2], p[1][3], x);
        P[0][3] = x[0]; P[1][3] = x[1]; P[2][3] = x[2];
      }
#pragma unroll
      for (int n = 0; n < NT; n += 2) {
        float t[2][4];
        cr_zero(t);
#pragma unroll
        for (int j = VP - 1; j >= 0; --j) {
          unsigned B[4];
          cr_ldm4t(vb + ((j * SUB + sb) * VS + n * 8) * 2, B);
#pragma unroll
          for (int i = 2 - j; i >= 0; --i) {
            cr_mma(t[0], P[i], B[0], B[1]);
            cr_mma(t[1], P[i], B[2], B[3]);
          }
        }
        if (b == rb && __any_sync(0xffffffffu, !cr_finite(t[0]) || !cr_finite(t[1]))) {
          // a value that is not finite met the zero weight of an earlier row: once more without such values, which then
          // go to their own row and the later ones
          cr_zero(t);
#pragma unroll
          for (int j = VP - 1; j >= 0; --j) {
            unsigned B[4];
            cr_ldm4t(vb + ((j * SUB + sb) * VS + n * 8) * 2, B);
#pragma unroll
            for (int i = 0; i < 4; ++i) B[i] = cr_finite_only(B[i]);
#pragma unroll
            for (int i = 2 - j; i >= 0; --i) {
              cr_mma(t[0], P[i], B[0], B[1]);
              cr_mma(t[1], P[i], B[2], B[3]);
            }
          }
#pragma unroll 1
          for (int s = 0; s < 16; ++s) {
            const float x0 = s & 8 ? (s & 1 ? p[1][1] : p[1][0]) : (s & 1 ? p[0][1] : p[0][0]);
            const float x1 = s & 8 ? (s & 1 ? p[1][3] : p[1][2]) : (s & 1 ? p[0][3] : p[0][2]);
            const float w0 = __shfl_sync(0xffffffffu, x0, (lane & 28) | ((s & 7) >> 1));
            const float w1 = __shfl_sync(0xffffffffu, x1, (lane & 28) | ((s & 7) >> 1));
#pragma unroll
            for (int j = 0; j < 2; ++j)
#pragma unroll
              for (int e = 0; e < 2; ++e) {
                const float v = __bfloat162float(Vs[(size_t)(sb + s) * VS + n0 + (n + j) * 8 + t4 * 2 + e]);
                if (fabsf(v) < INFINITY) continue;
                if (s <= g) t[j][e] = fmaf(w0, v, t[j][e]);
                if (s <= g + 8) t[j][e + 2] = fmaf(w1, v, t[j][e + 2]);
              }
          }
        }
        cr_add(acc[n], t[0]);
        cr_add(acc[n + 1], t[1]);
      }
    }
  }
  if (!work) return;
#pragma unroll
  for (int hi = 0; hi < 2; ++hi) {
    const int r = rb * 16 + g + 8 * hi;
    if (r >= live) continue;
    const size_t row = (size_t)(row0 + r);
    const float skip = MODE == kCrScan ? a.skip[head] : 0.f, factor = MODE == kCrDelta ? a.gates[(row * a.H + head) * 4 + 2] : 1.f;
    float* dst = a.out + row * a.H * a.V + (size_t)head * a.V + tile0 + n0 + t4 * 2;
    const __nv_bfloat16* x = a.v + row * a.ld + a.v0 + (size_t)head * a.V + tile0 + n0 + t4 * 2;
#pragma unroll
    for (int n = 0; n < NT; ++n) {
      float y0 = acc[n][2 * hi], y1 = acc[n][2 * hi + 1];
      if (MODE == kCrDelta) { y0 *= factor; y1 *= factor; }
      if (MODE == kCrScan) {
        const __nv_bfloat162 xx = *reinterpret_cast<const __nv_bfloat162*>(x + n * 8);
        y0 = fmaf(skip, __low2float(xx), y0);
        y1 = fmaf(skip, __high2float(xx), y1);
      }
      *reinterpret_cast<float2*>(dst + n * 8) = make_float2(y0, y1);
    }
  }
}

// VT: columns of a head an output CTA has.
template <int D, int VT, int Q, int SUB, int QKP, int VP, int MODE>
int launch_outputs(const CrArgs& a, int n_chunks, cudaStream_t stream) {
  constexpr size_t part_s = 3 * (size_t)VT * (D + kCrPad), part_kv = (size_t)QKP * SUB * (D + kCrPad) + (size_t)VP * SUB * (VT + kCrPad);
  constexpr size_t smem = ((size_t)QKP * Q * (D + kCrPad) + (part_s > part_kv ? part_s : part_kv)) * 2;
  static_assert(smem <= 220 * 1024, "shared memory of a chunk");
  static bool set = false;                // (the attribute is the function's: set twice by two threads, it is the same)
  if (!set) {
    const cudaError_t e = cudaFuncSetAttribute(chunk_output_kernel<D, VT, Q, SUB, QKP, VP, MODE>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    NF_REQUIRE(e == cudaSuccess, "chunk recurrence: cannot have %zu bytes of shared memory: %s", smem, cudaGetErrorString(e));
    set = true;
  }
  launch_chained(chunk_output_kernel<D, VT, Q, SUB, QKP, VP, MODE>, dim3(n_chunks, a.H, a.V / VT), dim3(kCrThreads), smem, stream, a);
  return check_launch("chunk_recurrence");
}

template <int D, int V, int VT, int Q, int SUB, int QKP, int VP, int MODE>
int launch_chunks(const CrArgs& a, int n_chunks, int n_runs, cudaStream_t stream) {
  constexpr size_t smem = ((size_t)QKP * Q * (D + kCrPad) + 3 * (size_t)Q * (V + kCrPad)) * 2;
  static_assert(smem <= 220 * 1024, "shared memory of a chunk");
  static bool set = false;
  if (!set) {
    const cudaError_t e = cudaFuncSetAttribute(chunk_state_kernel<D, V, Q, QKP, MODE>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    NF_REQUIRE(e == cudaSuccess, "chunk recurrence: cannot have %zu bytes of shared memory: %s", smem, cudaGetErrorString(e));
    set = true;
  }
  launch_chained(chunk_state_kernel<D, V, Q, QKP, MODE>, dim3(n_chunks, a.H), dim3(kCrThreads), smem, stream, a);
  launch_chained(chunk_chain_kernel<Q>, dim3(n_runs, a.H, (V * D / 4 + kCrThreads - 1) / kCrThreads), dim3(kCrThreads), 0, stream, a, V * D);
  return launch_outputs<D, VT, Q, SUB, QKP, VP, MODE>(a, n_chunks, stream);
}

// ---- the gated delta rule -------------------------------------------------------------------------------------------
//
//   S <- g_t S;  u_t = beta_t (v_t - S^T k_t);  S <- S + k_t u_t^T;  o_t = S^T q_t        (k_t, q_t unit vectors)
//
// Over a chunk, with A_t and D(s, t) as above and the chunk's inner products m_ts = beta_t D(s, t) k_s.k_t (s < t), the u
// solve a triangular system: U = T (V - [A_t k_t^T S_0]_t), T = (1 + m)^-1 diag(beta).  T depends on the keys and gates
// alone, so (1) makes it for all chunks and heads at once; (2) walks the chunks, a CTA a head and 16 value columns, with
// three products a chunk; (3) is the output kernel above with U for the values.  What the rows' norms scale (k and q are
// bfloat16 numbers over their norm) goes into the float32 factors, so that products with k and q stay exact.

constexpr int kDcRows = 64;               // rows a chunk

struct DcArgs {
  const __nv_bfloat16 *qkv, *ab;
  int ld, q0, k0, v0, ld_ab, a0, b0;
  const float *dt_bias, *A_log;
  float q_scale;
  int H, heads_per_group, V;
  CrChunks at;
  const int* seg_slot;
  float* state;
  long slot_stride;
  __nv_bfloat16* solve;                   // T as three parts: [n][H][3][64][64]
  float* coef;                            // [n][H][64][2]: A_t / |k_t|, D(t, end) / |k_t|
  float* gates;                           // [T][H][4]: g, 1 / |k|, q_scale / |q|, 0
  float* chunk_state;                     // [n][H][V][D]
  float* chunk_decay;                     // [n][H]
  float* u;                               // [T][H * V]
};

__device__ __forceinline__ void cr_cp16(void* dst, const void* src, bool ok) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(cr_smem(dst)), "l"(src), "r"(ok ? 16 : 0) : "memory");
}
__device__ __forceinline__ void cr_ldm2t(unsigned addr, unsigned& r0, unsigned& r1) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x2.trans.shared.b16 {%0,%1}, [%2];" : "=r"(r0), "=r"(r1) : "r"(addr) : "memory");
}

template <int D>
__global__ void __launch_bounds__(kCrThreads)
delta_chunk_solve_kernel(const DcArgs args) {
  constexpr int Q = kDcRows, KS = D + kCrPad, MS = Q + 4;
  extern __shared__ __align__(16) unsigned char cr_raw[];
  __nv_bfloat16* Ks = reinterpret_cast<__nv_bfloat16*>(cr_raw);              // [Q][KS]
  float* M = reinterpret_cast<float*>(Ks + Q * KS);                          // [Q][MS]
  __shared__ float s_g[Q], s_beta[Q], s_ik[Q], s_upto[Q], s_after[Q];
  __shared__ float s_diag[Q / 16][16][17];
  const int chunk = blockIdx.x, head = blockIdx.y, grp = head / args.heads_per_group;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  DcArgs a = args;
  const int2 place = cr_rows<Q>(a.at, chunk);
  const int row0 = place.x, live = place.y;
  chain_wait(a.qkv, a.ab);
  const __nv_bfloat16* kr = a.qkv + a.k0 + (size_t)grp * D;
  const __nv_bfloat16* qr = a.qkv + a.q0 + (size_t)grp * D;
  for (int r = warp; r < Q; r += kCrThreads / 32) {      // a warp a row: the key to shared memory, both norms
    float kk = 0.f, qq = 0.f;
    for (int c = lane * 4; c < D; c += 128) {
      float k[4] = {0.f, 0.f, 0.f, 0.f}, q[4] = {0.f, 0.f, 0.f, 0.f};
      uint2 raw = make_uint2(0, 0);
      if (r < live) {
        raw = *reinterpret_cast<const uint2*>(kr + (size_t)(row0 + r) * a.ld + c);
        load4(reinterpret_cast<const __nv_bfloat16*>(&raw), k);
        load4(qr + (size_t)(row0 + r) * a.ld + c, q);
      }
      *reinterpret_cast<uint2*>(Ks + r * KS + c) = raw;
#pragma unroll
      for (int e = 0; e < 4; ++e) { kk = fmaf(k[e], k[e], kk); qq = fmaf(q[e], q[e], qq); }
    }
    kk = warp_sum(kk);
    qq = warp_sum(qq);
    if (lane == 0) {
      float g = 1.f, beta = 0.f, ik = 0.f;
      if (r < live) {
        const __nv_bfloat16* ab = a.ab + (size_t)(row0 + r) * a.ld_ab;
        const float x = to_float(ab[a.a0 + head]) + a.dt_bias[head];
        g = expf(-expf(a.A_log[head]) * (fmaxf(x, 0.f) + log1pf(expf(-fabsf(x)))));
        beta = 1.f / (1.f + expf(-to_float(ab[a.b0 + head])));
        ik = 1.f / sqrtf(kk + 1e-6f);
        *reinterpret_cast<float4*>(a.gates + ((size_t)(row0 + r) * a.H + head) * 4) = make_float4(g, ik, a.q_scale / sqrtf(qq + 1e-6f), 0.f);
      }
      s_g[r] = g;
      s_beta[r] = beta;
      s_ik[r] = ik;
    }
  }
  __syncthreads();
  if (threadIdx.x < Q) cr_decay_table(s_g, threadIdx.x, s_upto, s_after, s_diag);
  __syncthreads();
  if (threadIdx.x < Q) {
    const int t = threadIdx.x, b = t >> 4;
    float before = 1.f, past = s_after[t];
    for (int x = 0; x < b; ++x) before *= s_upto[16 * x + 15];
    for (int x = b + 1; x < Q / 16; ++x) past *= s_upto[16 * x + 15];
    const float upto = before * s_upto[t];
    *reinterpret_cast<float2*>(a.coef + (((size_t)chunk * a.H + head) * Q + t) * 2) = make_float2(upto * s_ik[t], past * s_ik[t]);
    if (t == Q - 1) a.chunk_decay[(size_t)chunk * a.H + head] = upto;
  }
  {  // m_ts: warp w has rows 16 (w % 4) .. and columns 32 (w / 4) ..
    const int rb = warp & 3, c0 = (warp >> 2) * 32, g = lane >> 2, t4 = lane & 3, mat = lane >> 3, r8 = lane & 7;
    float p[4][4];
#pragma unroll
    for (int n = 0; n < 4; ++n)
#pragma unroll
      for (int e = 0; e < 4; ++e) p[n][e] = 0.f;
    const unsigned ka = cr_smem(Ks + (rb * 16 + (mat & 1) * 8 + r8) * KS + (mat >> 1) * 8);
    const unsigned kb = cr_smem(Ks + (c0 + (mat >> 1) * 8 + r8) * KS + (mat & 1) * 8);
    if (c0 <= rb * 16 + 15) {
#pragma unroll
      for (int k0 = 0; k0 < D; k0 += 16) {
        unsigned A[4], B[4];
        cr_ldm4(ka + k0 * 2, A);
#pragma unroll
        for (int n = 0; n < 4; n += 2) {
          cr_ldm4(kb + (n * 8 * KS + k0) * 2, B);
          float t[2][4];
          cr_zero(t);
          cr_mma(t[0], A, B[0], B[1]);
          cr_mma(t[1], A, B[2], B[3]);
          cr_add(p[n], t[0]);
          cr_add(p[n + 1], t[1]);
        }
      }
    }
#pragma unroll
    for (int n = 0; n < 4; ++n)
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const int s = c0 + n * 8 + t4 * 2 + (e & 1), t = rb * 16 + g + (e >> 1) * 8, b = s >> 4;
        float d = 0.f;
        if (s < t) {
          if (b == rb) d = s_diag[rb][s & 15][t & 15];
          else {
            d = s_after[s] * s_upto[t];
            for (int x = b + 1; x < rb; ++x) d *= s_upto[16 * x + 15];
          }
          d *= s_ik[s] * s_ik[t] * s_beta[t];
        }
        M[t * MS + s] = d == 0.f ? 0.f : d * p[n][e];
      }
  }
  __syncthreads();
  if (threadIdx.x < Q) {                 // thread j: column j of (1 + m)^-1 by forward substitution, times beta_j
    const int j = threadIdx.x;
    const float beta = s_beta[j];
    __nv_bfloat16* out = a.solve + ((size_t)chunk * a.H + head) * 3 * Q * Q + j;
    float x[Q];
#pragma unroll
    for (int t = 0; t < Q; ++t) x[t] = 0.f;
#pragma unroll
    for (int t = 0; t < Q; ++t) {
      float r[4] = {t == j ? 1.f : 0.f, 0.f, 0.f, 0.f};
#pragma unroll
      for (int s = 0; s < t; s += 4) {
        float m[4];
        load4(M + t * MS + s, m);
#pragma unroll
        for (int e = 0; e < 4; ++e) r[e] = fmaf(-m[e], x[s + e], r[e]);
      }
      x[t] = (r[0] + r[1]) + (r[2] + r[3]);
      float v = t < j ? 0.f : x[t] * beta;     // (also where beta is not a number)
#pragma unroll
      for (int i = 0; i < 3; ++i) {
        const __nv_bfloat16 h = __float2bfloat16_rn(v);
        out[(size_t)(i * Q + t) * Q] = h;
        v = isinf(__bfloat162float(h)) || isnan(__bfloat162float(h)) ? 0.f : v - __bfloat162float(h);
      }
    }
  }
}

// Two numbers' three parts to a place of three planes.
__device__ __forceinline__ void cr_put3(__nv_bfloat16* dst, size_t plane, float x, float y) {
  unsigned p[3];
  cr_split<3>(x, y, p);
#pragma unroll
  for (int i = 0; i < 3; ++i) *reinterpret_cast<unsigned*>(dst + i * plane) = p[i];
}

template <int D>
__global__ void __launch_bounds__(kCrThreads)
delta_chunk_chain_kernel(const DcArgs args) {
  constexpr int Q = kDcRows, KS = D + kCrPad, TS = Q + kCrPad, XS = 16 + kCrPad, NT = D / 64;
  extern __shared__ __align__(16) unsigned char cr_raw[];
  __nv_bfloat16* Ks = reinterpret_cast<__nv_bfloat16*>(cr_raw);              // [2][Q][KS]
  __nv_bfloat16* Ts = Ks + 2 * Q * KS;                                       // [2][3][Q][TS]
  __nv_bfloat16* Vs = Ts + 2 * 3 * Q * TS;                                   // [2][Q][16]
  __nv_bfloat16* Ss = Vs + 2 * Q * 16;                                       // [3][16][KS]
  __nv_bfloat16* Xs = Ss + 3 * 16 * KS;                                      // [3][Q][XS]
  __nv_bfloat16* Us = Xs + 3 * Q * XS;                                       // [3][Q][XS]
  float* coef = reinterpret_cast<float*>(Us + 3 * Q * XS);                   // [2][Q][2]
  const int run = blockIdx.x, head = blockIdx.y, v0 = blockIdx.z * 16, grp = head / args.heads_per_group;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int g = lane >> 2, t4 = lane & 3, mat = lane >> 3, r8 = lane & 7;
  DcArgs a = args;
  const CrPlace place = cr_find<Q, true>(a.at, a.at.first_run + run);
  const int3 own = cr_run<Q>(a.at, place);
  const int seg = place.seg, first = own.x, n = own.y, seg_row = place.row0 + own.z * Q, seg_rows = place.rows - own.z * Q;
  chain_wait(a.qkv, a.solve, a.coef, a.chunk_decay, a.state);
  auto fetch = [&](int c) {
    if (c < n) {
      const int b = c & 1, chunk = first + c, row0 = seg_row + c * Q, live = min(Q, seg_rows - c * Q);
      const __nv_bfloat16* kr = a.qkv + (size_t)row0 * a.ld + a.k0 + (size_t)grp * D;
#pragma unroll
      for (int i = threadIdx.x; i < Q * (D / 8); i += kCrThreads) {
        const int r = i / (D / 8), col = (i % (D / 8)) * 8;
        cr_cp16(Ks + (b * Q + r) * KS + col, r < live ? kr + (size_t)r * a.ld + col : a.qkv, r < live);
      }
      const __nv_bfloat16* tp = a.solve + ((size_t)chunk * a.H + head) * 3 * Q * Q;
#pragma unroll
      for (int i = threadIdx.x; i < 3 * Q * (Q / 8); i += kCrThreads)
        cr_cp16(Ts + (b * 3 * Q + i / (Q / 8)) * TS + (i % (Q / 8)) * 8, tp + (size_t)i * 8, true);
      if (threadIdx.x < Q * 2) {
        const int r = threadIdx.x >> 1, col = (threadIdx.x & 1) * 8;
        const __nv_bfloat16* vr = a.qkv + (size_t)(row0 + r) * a.ld + a.v0 + (size_t)head * a.V + v0 + col;
        cr_cp16(Vs + (b * Q + r) * 16 + col, r < live ? vr : a.qkv, r < live);
      } else if (threadIdx.x < Q * 2 + Q / 2) {
        const int i = threadIdx.x - Q * 2;
        cr_cp16(coef + b * Q * 2 + i * 4, a.coef + ((size_t)chunk * a.H + head) * Q * 2 + i * 4, true);
      }
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  fetch(0);
  // the state: value columns g and g + 8 of the sixteen, key dimensions of this warp's D / 8
  const int d0 = warp * (D / 8) + 2 * t4;
  float* slot = a.state + (size_t)a.seg_slot[seg] * a.slot_stride + ((size_t)head * a.V + v0 + g) * D + d0;
  float s[NT][4];
#pragma unroll
  for (int i = 0; i < NT; ++i) {
    const float2 x = *reinterpret_cast<const float2*>(slot + 8 * i), y = *reinterpret_cast<const float2*>(slot + 8 * D + 8 * i);
    s[i][0] = x.x; s[i][1] = x.y; s[i][2] = y.x; s[i][3] = y.y;
    cr_put3(Ss + g * KS + d0 + 8 * i, 16 * KS, s[i][0], s[i][1]);
    cr_put3(Ss + (g + 8) * KS + d0 + 8 * i, 16 * KS, s[i][2], s[i][3]);
  }
  const int mt = warp & 3, nt = warp >> 2;           // rows 16 mt .., columns 8 nt .. of the first two products
  const int tr = mt * 16 + g, col = nt * 8 + 2 * t4;
  for (int c = 0; c < n; ++c) {
    const int b = c & 1, chunk = first + c, row0 = seg_row + c * Q, live = min(Q, seg_rows - c * Q);
    const float decay = a.chunk_decay[(size_t)chunk * a.H + head];
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    __syncthreads();                                 // the chunk is in; the state's parts are written; the rest is free
    fetch(c + 1);
    float* start = a.chunk_state + (((size_t)chunk * a.H + head) * a.V + v0 + g) * D + d0;
#pragma unroll
    for (int i = 0; i < NT; ++i) {
      *reinterpret_cast<float2*>(start + 8 * i) = make_float2(s[i][0], s[i][1]);
      *reinterpret_cast<float2*>(start + 8 * D + 8 * i) = make_float2(s[i][2], s[i][3]);
    }
    const __nv_bfloat16* K = Ks + b * Q * KS;
    {  // x_t = v_t - A_t S^T k_t
      float y[1][4];
      cr_zero(y);
      const unsigned ka = cr_smem(K + (mt * 16 + (mat & 1) * 8 + r8) * KS + (mat >> 1) * 8);
      const unsigned sb = cr_smem(Ss + (nt * 8 + r8) * KS + mat * 8);
#pragma unroll
      for (int k0 = 0; k0 < D; k0 += 32) {
        unsigned A0[4], A1[4], B[4];
        cr_ldm4(ka + k0 * 2, A0);
        cr_ldm4(ka + (k0 + 16) * 2, A1);
        float t[2][4];
        cr_zero(t);
#pragma unroll
        for (int i = 2; i >= 0; --i) {
          cr_ldm4(sb + (i * 16 * KS + k0) * 2, B);
          cr_mma(t[0], A0, B[0], B[1]);
          cr_mma(t[1], A1, B[2], B[3]);
        }
        cr_add(y[0], t[0]);
        cr_add(y[0], t[1]);
      }
      const float c0 = coef[(b * Q + tr) * 2], c1 = coef[(b * Q + tr + 8) * 2];
      const __nv_bfloat162 va = *reinterpret_cast<const __nv_bfloat162*>(Vs + (b * Q + tr) * 16 + col);
      const __nv_bfloat162 vb = *reinterpret_cast<const __nv_bfloat162*>(Vs + (b * Q + tr + 8) * 16 + col);
      cr_put3(Xs + tr * XS + col, Q * XS, __low2float(va) - c0 * y[0][0], __high2float(va) - c0 * y[0][1]);
      cr_put3(Xs + (tr + 8) * XS + col, Q * XS, __low2float(vb) - c1 * y[0][2], __high2float(vb) - c1 * y[0][3]);
    }
    __syncthreads();
    {  // U = T X
      float u[1][4];
      cr_zero(u);
      const unsigned ta = cr_smem(Ts + (b * 3 * Q + mt * 16 + (mat & 1) * 8 + r8) * TS + (mat >> 1) * 8);
      const unsigned xb = cr_smem(Xs + (lane & 15) * XS + nt * 8);
      // u += the sixteen ks of T times X; apart: the values of X that are not finite are left out
      auto add_sixteen = [&](int ks, bool apart) {
        unsigned A[3][4], B[3][2];
#pragma unroll
        for (int i = 0; i < 3; ++i) {
          cr_ldm4(ta + (i * Q * TS + ks * 16) * 2, A[i]);
          cr_ldm2t(xb + ((i * Q + ks * 16) * XS) * 2, B[i][0], B[i][1]);
          if (apart) {
            B[i][0] = cr_finite_only(B[i][0]);
            B[i][1] = cr_finite_only(B[i][1]);
          }
        }
        float t[3][4];                             // (three chains side by side: this is the walk from chunk to chunk)
        cr_zero(t);
        cr_mma(t[2], A[0], B[2][0], B[2][1]);
        cr_mma(t[1], A[0], B[1][0], B[1][1]);
        cr_mma(t[0], A[0], B[0][0], B[0][1]);
        cr_mma(t[2], A[1], B[1][0], B[1][1]);
        cr_mma(t[1], A[1], B[0][0], B[0][1]);
        cr_mma(t[2], A[2], B[0][0], B[0][1]);
#pragma unroll
        for (int e = 0; e < 4; ++e) u[0][e] += t[0][e] + (t[1][e] + t[2][e]);
      };
      for (int ks = 0; ks <= mt; ++ks) add_sixteen(ks, false);
      if (__any_sync(0xffffffffu, !cr_finite(u[0]))) {                       // (see the outputs)
        cr_zero(u);
#pragma unroll 1
        for (int ks = 0; ks <= mt; ++ks) add_sixteen(ks, ks == mt);
        auto whole = [&](const __nv_bfloat16* x) {
          return (__bfloat162float(x[0]) + __bfloat162float(x[Q * TS])) + __bfloat162float(x[2 * Q * TS]);
        };
        const __nv_bfloat16* tp = Ts + ((size_t)b * 3 * Q + tr) * TS + mt * 16;
#pragma unroll 1
        for (int j = 0; j < 16; ++j)
#pragma unroll
          for (int e = 0; e < 2; ++e) {
            const float x = __bfloat162float(Xs[(mt * 16 + j) * XS + col + e]);
            if (fabsf(x) < INFINITY) continue;
            if (j <= g) u[0][e] = fmaf(whole(tp + j), x, u[0][e]);
            if (j <= g + 8) u[0][e + 2] = fmaf(whole(tp + 8 * TS + j), x, u[0][e + 2]);
          }
      }
      float* dst = a.u + (size_t)(row0 + tr) * a.H * a.V + (size_t)head * a.V + v0 + col;
      if (tr < live) *reinterpret_cast<float2*>(dst) = make_float2(u[0][0], u[0][1]);
      if (tr + 8 < live) *reinterpret_cast<float2*>(dst + (size_t)8 * a.H * a.V) = make_float2(u[0][2], u[0][3]);
      const float c0 = coef[(b * Q + tr) * 2 + 1], c1 = coef[(b * Q + tr + 8) * 2 + 1];
      cr_put3(Us + tr * XS + col, Q * XS, u[0][0] * c0, u[0][1] * c0);
      cr_put3(Us + (tr + 8) * XS + col, Q * XS, u[0][2] * c1, u[0][3] * c1);
    }
    __syncthreads();
    {  // S = A S + sum_t D(t, end) u_t k_t^T
      float w[NT][4];
      cr_zero(w);
      const unsigned ua = cr_smem(Us + ((mat >> 1) * 8 + r8) * XS + (mat & 1) * 8);
      const unsigned kb = cr_smem(K + ((mat & 1) * 8 + r8) * KS + warp * (D / 8) + (NT == 2 ? (mat >> 1) * 8 : 0));
#pragma unroll
      for (int ks = 0; ks < Q / 16; ++ks) {
        unsigned A[3][4], B[4];
        float t[NT][4];
        cr_zero(t);
        cr_ldm4t(kb + ks * 16 * KS * 2, B);          // (one column tile: the third and fourth repeat the first two)
#pragma unroll
        for (int i = 2; i >= 0; --i) {
          cr_ldm4t(ua + (i * Q + ks * 16) * XS * 2, A[i]);
#pragma unroll
          for (int j = 0; j < NT; ++j) cr_mma(t[j], A[i], B[2 * j], B[2 * j + 1]);
        }
#pragma unroll
        for (int j = 0; j < NT; ++j) cr_add(w[j], t[j]);
      }
#pragma unroll
      for (int j = 0; j < NT; ++j) {
#pragma unroll
        for (int e = 0; e < 4; ++e) s[j][e] = fmaf(decay, s[j][e], w[j][e]);
        cr_put3(Ss + g * KS + d0 + 8 * j, 16 * KS, s[j][0], s[j][1]);
        cr_put3(Ss + (g + 8) * KS + d0 + 8 * j, 16 * KS, s[j][2], s[j][3]);
      }
    }
  }
#pragma unroll
  for (int i = 0; i < NT; ++i) {
    *reinterpret_cast<float2*>(slot + 8 * i) = make_float2(s[i][0], s[i][1]);
    *reinterpret_cast<float2*>(slot + 8 * D + 8 * i) = make_float2(s[i][2], s[i][3]);
  }
}

template <int D>
int launch_delta(const DcArgs& d, const CrArgs& a, int n_chunks, int n_runs, cudaStream_t stream) {
  constexpr int Q = kDcRows;
  constexpr size_t smem1 = (size_t)Q * (D + kCrPad) * 2 + (size_t)Q * (Q + 4) * 4;
  constexpr size_t smem2 = ((size_t)2 * Q * (D + kCrPad) + 6 * Q * (Q + kCrPad) + 2 * Q * 16 + 3 * 16 * (D + kCrPad) + 6 * Q * (16 + kCrPad)) * 2 + 2 * Q * 2 * 4;
  static bool set = false;
  if (!set) {
    cudaError_t e = cudaFuncSetAttribute(delta_chunk_solve_kernel<D>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem1);
    if (e == cudaSuccess) e = cudaFuncSetAttribute(delta_chunk_chain_kernel<D>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem2);
    NF_REQUIRE(e == cudaSuccess, "delta rule: cannot have %zu and %zu bytes of shared memory: %s", smem1, smem2, cudaGetErrorString(e));
    set = true;
  }
  launch_chained(delta_chunk_solve_kernel<D>, dim3(n_chunks, d.H), dim3(kCrThreads), smem1, stream, d);
  launch_chained(delta_chunk_chain_kernel<D>, dim3(n_runs, d.H, d.V / 16), dim3(kCrThreads), smem2, stream, d);
  return launch_outputs<D, 64, Q, 32, 1, 3, kCrDelta>(a, n_chunks, stream);
}

}  // namespace
}  // namespace nf

using namespace nf;

// Rows a chunk; 0: these sizes are not served here.  scan: the selective scan, else linear attention.
extern "C" int nf_chunk_recurrence_rows(int D, int V, int scan) {
  if (scan) return (D == 64 || D == 128) && V == 64 ? 128 : 0;
  return (D == 64 || D == 128) && V == 128 ? 64 : 0;
}

// The selective scan of chunks first_chunk .. + n_chunks of the segments of at least min_rows rows (counted over all such
// segments, nf_chunk_recurrence_rows rows each but a segment's last); they belong to n_runs of those segments, from number
// first_run on.  Arguments as nf_ssd_scan's (bfloat16).  chunk_state float32 [n_chunks, heads, P, N], chunk_decay float32 [n_chunks, heads]: scratch.
extern "C" int nf_chunk_scan(const void* xbc, int ldx, int x0, int b0, int c0, const void* dt, int ld_dt, int dt0,
                             const float* dt_bias, const float* A_log, const float* skip, float* state, long long slot_stride,
                             const int* seg_slot, const int* seg_row0, int S, int min_rows, int first_chunk, int n_chunks, int first_run, int n_runs,
                             float* chunk_state, float* chunk_decay, float* out, int heads, int P, int N, int groups,
                             cudaStream_t stream) {
  if (n_chunks == 0) return 0;
  NF_REQUIRE(nf_chunk_recurrence_rows(N, P, 1) > 0 && groups > 0 && heads % groups == 0 && heads <= 65535, "chunk scan: sizes N=%d P=%d heads=%d", N, P, heads);
  NF_REQUIRE(ldx % 8 == 0 && x0 % 8 == 0 && b0 % 8 == 0 && c0 % 8 == 0 && (uintptr_t)xbc % 16 == 0 && slot_stride % 4 == 0 &&
             (uintptr_t)state % 16 == 0 && (uintptr_t)out % 16 == 0, "chunk scan: rows and states must be 16-byte aligned");
  CrArgs a = {};
  a.q = a.k = a.v = (const __nv_bfloat16*)xbc;
  a.ld = ldx; a.q0 = c0; a.k0 = b0; a.v0 = x0;
  a.H = heads; a.heads_per_group = heads / groups; a.V = P;
  a.dt = (const __nv_bfloat16*)dt; a.ld_dt = ld_dt; a.dt0 = dt0;
  a.dt_bias = dt_bias; a.A_log = A_log; a.skip = skip;
  a.at = {seg_row0, S, min_rows, first_chunk, n_chunks, first_run}; a.seg_slot = seg_slot;
  a.state = state; a.slot_stride = (long)slot_stride;
  a.chunk_state = chunk_state; a.chunk_decay = chunk_decay; a.out = out;
  if (N == 128) return launch_chunks<128, 64, 64, 128, 64, 1, 1, kCrScan>(a, n_chunks, n_runs, stream);
  return launch_chunks<64, 64, 64, 128, 64, 1, 1, kCrScan>(a, n_chunks, n_runs, stream);
}

// Linear attention of such chunks: prepared float32 [T, 2, H, D] (q and k), v bfloat16 [T, ld] from v0 on
// (through SiLU with v_silu), decay float32 [H]; the rest as above.
extern "C" int nf_chunk_linear_attention(const float* prepared, const void* v, int ld, int v0, int v_silu, const float* decay,
                                         float* state, long long slot_stride, const int* seg_slot,
                                         const int* seg_row0, int S, int min_rows, int first_chunk, int n_chunks,
                                         int first_run, int n_runs, float* chunk_state,
                                         float* chunk_decay, float* out, int H, int D, int V, cudaStream_t stream) {
  if (n_chunks == 0) return 0;
  NF_REQUIRE(nf_chunk_recurrence_rows(D, V, 0) > 0 && H > 0 && H <= 65535 && decay, "chunk linear attention: sizes D=%d V=%d H=%d", D, V, H);
  NF_REQUIRE(ld % 8 == 0 && v0 % 8 == 0 && (uintptr_t)v % 16 == 0 && (uintptr_t)prepared % 16 == 0 && slot_stride % 4 == 0 &&
             (uintptr_t)state % 16 == 0 && (uintptr_t)out % 16 == 0, "chunk linear attention: rows and states must be 16-byte aligned");
  CrArgs a = {};
  a.v = (const __nv_bfloat16*)v;
  a.ld = ld; a.v0 = v0; a.v_silu = v_silu; a.prepared = prepared;
  a.H = H; a.heads_per_group = 1; a.V = V;
  a.decay = decay;
  a.at = {seg_row0, S, min_rows, first_chunk, n_chunks, first_run}; a.seg_slot = seg_slot;
  a.state = state; a.slot_stride = (long)slot_stride;
  a.chunk_state = chunk_state; a.chunk_decay = chunk_decay; a.out = out;
  if (D == 128) return v_silu ? launch_chunks<128, 128, 64, 64, 32, 3, 3, kCrDecay>(a, n_chunks, n_runs, stream)
                              : launch_chunks<128, 128, 64, 64, 32, 3, 1, kCrDecay>(a, n_chunks, n_runs, stream);
  return v_silu ? launch_chunks<64, 128, 128, 64, 32, 3, 3, kCrDecay>(a, n_chunks, n_runs, stream)
                : launch_chunks<64, 128, 128, 64, 32, 3, 1, kCrDecay>(a, n_chunks, n_runs, stream);
}

extern "C" int nf_chunk_delta_rule_rows(int D, int V) { return (D == 64 || D == 128) && V % 64 == 0 ? kDcRows : 0; }

// The gated delta rule of such chunks; arguments as nf_delta_rule's (bfloat16).  Scratch: solve bfloat16
// [n_chunks, H, 3, 64, 64], coef float32 [n_chunks, H, 64, 2], gates float32 [T, H, 4], u float32 [T, H * V], chunk_state
// float32 [n_chunks, H, V, D], chunk_decay float32 [n_chunks, H].
extern "C" int nf_chunk_delta_rule(const void* qkv, int ld, int q0, int k0, int v0, const void* ab, int ld_ab, int a0, int b0,
                                   const float* dt_bias, const float* A_log, float q_scale, float* state, long long slot_stride,
                                   const int* seg_slot, const int* seg_row0, int S, int min_rows, int first_chunk, int n_chunks,
                                   int first_run, int n_runs, void* solve,
                                   float* coef, float* gates, float* u, float* chunk_state, float* chunk_decay, float* out,
                                   int H, int G, int D, int V, cudaStream_t stream) {
  if (n_chunks == 0) return 0;
  NF_REQUIRE(nf_chunk_delta_rule_rows(D, V) > 0 && G > 0 && H > 0 && H % G == 0 && H <= 65535, "chunk delta rule: sizes D=%d V=%d H=%d G=%d", D, V, H, G);
  NF_REQUIRE(ld % 8 == 0 && q0 % 8 == 0 && k0 % 8 == 0 && v0 % 8 == 0 && (uintptr_t)qkv % 16 == 0 && slot_stride % 4 == 0 &&
             (uintptr_t)state % 16 == 0 && (uintptr_t)out % 16 == 0, "chunk delta rule: rows and states must be 16-byte aligned");
  DcArgs d = {};
  d.qkv = (const __nv_bfloat16*)qkv; d.ab = (const __nv_bfloat16*)ab;
  d.ld = ld; d.q0 = q0; d.k0 = k0; d.v0 = v0; d.ld_ab = ld_ab; d.a0 = a0; d.b0 = b0;
  d.dt_bias = dt_bias; d.A_log = A_log; d.q_scale = q_scale;
  d.H = H; d.heads_per_group = H / G; d.V = V;
  d.at = {seg_row0, S, min_rows, first_chunk, n_chunks, first_run}; d.seg_slot = seg_slot;
  d.state = state; d.slot_stride = (long)slot_stride;
  d.solve = (__nv_bfloat16*)solve; d.coef = coef; d.gates = gates;
  d.chunk_state = chunk_state; d.chunk_decay = chunk_decay; d.u = u;
  CrArgs a = {};
  a.q = a.k = d.qkv;
  a.ld = ld; a.q0 = q0; a.k0 = k0;
  a.H = H; a.heads_per_group = H / G; a.V = V;
  a.values = u; a.gates = gates;
  a.at = d.at; a.chunk_state = chunk_state; a.out = out;
  return D == 128 ? launch_delta<128>(d, a, n_chunks, n_runs, stream) : launch_delta<64>(d, a, n_chunks, n_runs, stream);
}
