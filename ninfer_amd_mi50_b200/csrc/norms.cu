// Row-wise kernels beside those of elementwise.cu: a layer norm (mean taken off, weight, no
// bias) fused with the residual sum; an RMS norm of a column slice; the gated RMS norm in
// equal parts that follows a state-space mixer; a vector added to every row of the stream; a
// sigmoid gate; rows gathered in the experts' order and scaled by their routing weight.
//
// All statistics are float32 whatever the activations' type.  The layer norm's variance is the
// mean of the squared deviations from the mean (two passes over a row kept in shared memory),
// not E[x^2] - mean^2.
#define NF_CHAIN_CLASS 2
#include "common.cuh"

namespace nf {

// h[t] += delta[t] (if delta); out[t] = (h[t] - mean) * rsqrt(var + eps) * w.
// With `rows`, row r reads h[rows[r]] / delta[rows[r]], writes out[r] and leaves h alone.
// With `y`, delta[t] is the routed experts' sum that was left pending,
// sum_j wts[t, j] * y[inv[t * k + j]] (j ascending; wts null: unit weights), rounded to T as the
// separate combine kernel rounds it, so both ways give the same bits.
// VEC: the row's width is a multiple of 4 and every operand's rows start on 16 bytes (8 for bfloat16): a thread
// owns runs of four consecutive elements and moves each run in one access.  Which elements a thread owns, and the
// order in which it adds them up, is the same whether the sum that is added comes from `delta` or from `y`.
template <typename T, bool GATHER, bool VEC>
__global__ void add_layernorm_kernel(float* __restrict__ h, const T* __restrict__ delta,
                                     const int* __restrict__ rows, const float* __restrict__ w,
                                     float eps, T* __restrict__ out, int hidden, const T* __restrict__ y,
                                     const int* __restrict__ inv, const float* __restrict__ wts, int k) {
  extern __shared__ __align__(16) float row[];      // [hidden]
  __shared__ float red[33];
  const int r = blockIdx.x;
  constexpr int W = VEC ? 4 : 1;
  const int units = hidden / W;
  chain_release_if_small();
  // the weights of this thread's first run (all of them up to 4 * blockDim numbers) are asked for before the wait
  float4 w_first = make_float4(0.f, 0.f, 0.f, 0.f);
  if (VEC && (int)threadIdx.x < units) w_first = *reinterpret_cast<const float4*>(w + threadIdx.x * 4);
  chain_wait(h, delta, rows, y, inv, wts);
  const int src = GATHER ? rows[r] : r;
  float* hr = h + (size_t)src * hidden;
  const T* dr = delta ? delta + (size_t)src * hidden : nullptr;
  T* o = out + (size_t)r * hidden;
  float s = 0.f;
  for (int u = threadIdx.x; u < units; u += blockDim.x) {
    const int i = u * W;
    float v[W];
    if constexpr (VEC) {
      const float4 hv = *reinterpret_cast<const float4*>(hr + i);
      v[0] = hv.x; v[1] = hv.y; v[2] = hv.z; v[3] = hv.w;
    } else {
      v[0] = hr[i];
    }
    if (y) {
      float acc[W];
#pragma unroll
      for (int e = 0; e < W; ++e) acc[e] = 0.f;
      for (int j = 0; j < k; ++j) {
        const float wt = wts ? wts[(size_t)src * k + j] : 1.f;
        const T* yr = y + (size_t)inv[(size_t)src * k + j] * hidden + i;
        float yv[W];
        if constexpr (VEC) load4(yr, yv); else yv[0] = to_float(yr[0]);
#pragma unroll
        for (int e = 0; e < W; ++e) acc[e] += wt * yv[e];
      }
#pragma unroll
      for (int e = 0; e < W; ++e) v[e] += to_float(from_float<T>(acc[e]));
    } else if (dr) {
      float dv[W];
      if constexpr (VEC) load4(dr + i, dv); else dv[0] = to_float(dr[i]);
#pragma unroll
      for (int e = 0; e < W; ++e) v[e] += dv[e];
    }
    if (!GATHER && (y || dr)) {
      if constexpr (VEC) *reinterpret_cast<float4*>(hr + i) = make_float4(v[0], v[1], v[2], v[3]);
      else hr[i] = v[0];
    }
#pragma unroll
    for (int e = 0; e < W; ++e) { row[i + e] = v[e]; s += v[e]; }
  }
  const float mean = block_sum(s, red) / (float)hidden;
  float ss = 0.f;
  for (int u = threadIdx.x; u < units; u += blockDim.x) {
#pragma unroll
    for (int e = 0; e < W; ++e) {
      const float d = row[u * W + e] - mean;
      ss += d * d;
    }
  }
  const float rstd = rsqrtf(block_sum(ss, red) / (float)hidden + eps);
  for (int u = threadIdx.x; u < units; u += blockDim.x) {
    const int i = u * W;
    if constexpr (VEC) {
      const float4 wv = u == (int)threadIdx.x ? w_first : *reinterpret_cast<const float4*>(w + i);
      const float ov[4] = {(row[i] - mean) * rstd * wv.x, (row[i + 1] - mean) * rstd * wv.y,
                           (row[i + 2] - mean) * rstd * wv.z, (row[i + 3] - mean) * rstd * wv.w};
      store4(o + i, ov);
    } else {
      o[i] = from_float<T>((row[i] - mean) * rstd * w[i]);
    }
  }
}

// The same for rows of up to 8,192 numbers in runs of four, all rows in place (no list, no pending sum): the row in
// registers, rows walked as `row_ctas` gives them out.  Same sums in the same order.
template <typename T, int R, bool WALK>
__global__ void __launch_bounds__(512)
add_layernorm_regs_kernel(float* __restrict__ h, const T* __restrict__ delta, const float* __restrict__ w, float eps,
                          T* __restrict__ out, int hidden, int rows) {
  __shared__ float red[33];
  chain_release_if_small();
  float wk[R][4], v[R][4], hn[R][4], dn[R][4];
#pragma unroll
  for (int c = 0; c < R; ++c) {
    const int i = (c * blockDim.x + threadIdx.x) * 4;
    if (i < hidden) load4(w + i, wk[c]);
  }
  chain_wait(h, delta);
  auto ask = [&](int r) {
#pragma unroll
    for (int c = 0; c < R; ++c) {
      const int i = (c * blockDim.x + threadIdx.x) * 4;
      if (i < hidden) {
        load4(h + (size_t)r * hidden + i, hn[c]);
        if (delta) load4(delta + (size_t)r * hidden + i, dn[c]);
      }
    }
  };
  ask(blockIdx.x);
  for (int r = blockIdx.x; r < rows; r += gridDim.x) {
    float s = 0.f;
#pragma unroll
    for (int c = 0; c < R; ++c) {
      const int i = (c * blockDim.x + threadIdx.x) * 4;
      if (i >= hidden) continue;
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        v[c][e] = hn[c][e];
        if (delta) v[c][e] += dn[c][e];
        s += v[c][e];
      }
      if (delta) store4(h + (size_t)r * hidden + i, v[c]);
    }
    if (WALK && r + (int)gridDim.x < rows) ask(r + gridDim.x);
    const float mean = block_sum(s, red) / (float)hidden;
    float ss = 0.f;
#pragma unroll
    for (int c = 0; c < R; ++c)
      if ((c * (int)blockDim.x + (int)threadIdx.x) * 4 < hidden) {
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const float d = v[c][e] - mean;
          ss += d * d;
        }
      }
    const float rstd = rsqrtf(block_sum(ss, red) / (float)hidden + eps);
#pragma unroll
    for (int c = 0; c < R; ++c) {
      const int i = (c * blockDim.x + threadIdx.x) * 4;
      if (i >= hidden) continue;
      float o[4];
#pragma unroll
      for (int e = 0; e < 4; ++e) o[e] = (v[c][e] - mean) * rstd * wk[c][e];
      store4(out + (size_t)r * hidden + i, o);
    }
    if (!WALK) return;
  }
}

// RMS norm in `groups` equal consecutive parts, fused with the residual sum of up to two contributions (a
// mixer's and a feed-forward's that ran side by side):
//   h[t] += d1[t] (+ d2[t]);  out[t] = part / sqrt(mean(part^2) + eps) * w   for each part of h[t].
// With `rows`, row r reads h[rows[r]] / d1[rows[r]] / d2[rows[r]], writes out[r] and leaves h alone.
// The row waits in shared memory between the passes; warps are dealt out evenly to the groups.
// VEC: a group is a multiple of 4 elements and every operand's rows are aligned: runs of four an access.
template <typename T, bool GATHER, bool VEC>
__global__ void __launch_bounds__(256)
add_group_rmsnorm_kernel(float* __restrict__ h, const T* __restrict__ d1, const T* __restrict__ d2,
                         const int* __restrict__ rows, const float* __restrict__ w, float eps, int groups,
                         T* __restrict__ out, int hidden) {
  extern __shared__ __align__(16) float row[];      // [hidden], then partial sums [groups][warps a group], then inv [groups]
  const int r = blockIdx.x;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nwarp = blockDim.x >> 5;
  const int gs = hidden / groups;
  const int wpg = nwarp > groups ? nwarp / groups : 1;      // warps a group
  float* part = row + hidden;
  float* inv = part + groups * wpg;
  constexpr int W = VEC ? 4 : 1;
  chain_release_if_small();
  chain_wait(h, d1, d2, rows);
  const int src = GATHER ? rows[r] : r;
  float* hr = h + (size_t)src * hidden;
  const T* a = d1 ? d1 + (size_t)src * hidden : nullptr;
  const T* b = d2 ? d2 + (size_t)src * hidden : nullptr;
  for (int i = threadIdx.x * W; i < hidden; i += blockDim.x * W) {
    float v[W], x[W];
    if constexpr (VEC) load4(hr + i, v); else v[0] = hr[i];
    if (a) {
      if constexpr (VEC) load4(a + i, x); else x[0] = to_float(a[i]);
#pragma unroll
      for (int e = 0; e < W; ++e) v[e] += x[e];
    }
    if (b) {
      if constexpr (VEC) load4(b + i, x); else x[0] = to_float(b[i]);
#pragma unroll
      for (int e = 0; e < W; ++e) v[e] += x[e];
    }
    if (!GATHER && (a || b)) {
      if constexpr (VEC) store4(hr + i, v); else hr[i] = v[0];
    }
#pragma unroll
    for (int e = 0; e < W; ++e) row[i + e] = v[e];
  }
  __syncthreads();
  for (int g = warp / wpg; g < groups; g += (nwarp + wpg - 1) / wpg) {
    const int sub = warp - (warp / wpg) * wpg;
    float ss = 0.f;
    for (int i = (sub * 32 + lane) * W; i < gs; i += wpg * 32 * W) {
      float v[W];
      if constexpr (VEC) load4(row + g * gs + i, v); else v[0] = row[g * gs + i];
#pragma unroll
      for (int e = 0; e < W; ++e) ss = fmaf(v[e], v[e], ss);
    }
    ss = warp_sum(ss);
    if (lane == 0) part[g * wpg + sub] = ss;
  }
  __syncthreads();
  for (int g = threadIdx.x; g < groups; g += blockDim.x) {
    float ss = 0.f;
    for (int s = 0; s < wpg; ++s) ss += part[g * wpg + s];
    inv[g] = 1.f / sqrtf(ss / (float)gs + eps);
  }
  __syncthreads();
  T* o = out + (size_t)r * hidden;
  for (int i = threadIdx.x * W; i < hidden; i += blockDim.x * W) {
    const float f = inv[i / gs];
    if constexpr (VEC) {
      float v[4], wv[4];
      load4(row + i, v);
      load4(w + i, wv);
#pragma unroll
      for (int e = 0; e < 4; ++e) v[e] = v[e] * f * wv[e];
      store4(o + i, v);
    } else {
      o[i] = from_float<T>(row[i] * f * w[i]);
    }
  }
}

// The row-wise norms below in their wide form: a thread owns R runs of four consecutive elements of a row's part, keeps
// them in registers between the two passes and asks for the weights, which no kernel writes, before the wait.  In a decode
// step such a kernel is a chain of trips to memory (rows of 2,048 and 4,096 read element by element, twice, with the weight
// last, took 6 to 10 us, now 3 to 5), in a prompt it moves each row once.  Four layers of 2,048, prompts of 900 to 2,048 tokens and 16
// decoded ones: latent attention and scans 5.43 -> 5.09 ms, linear and windowed attention 6.93 -> 6.28, attention beside
// scans and delta rules 10.87 -> 10.55.
// MODE 0: out = x / rms(x) * w.  1: x = y * silu(z), out = x / rms(x) * w.  2, 3: out = y / rms(y) * w * act(z), act the
// silu or the sigmoid.  blockIdx.y: the part of the row.
template <typename TY, typename TZ, typename T, int R, int MODE, bool WALK>
__global__ void __launch_bounds__(512)
part_norm_vec_kernel(const TY* __restrict__ y, int ldy, int ycol0, const TZ* __restrict__ zsrc, int ldz, int zcol0,
                     const float* __restrict__ w, float eps, T* __restrict__ out, int ldo, int n, int rows) {
  __shared__ float red[33];
  const int c0 = blockIdx.y * n;
  chain_release_if_small();
  float wk[R][4], v[R][4], z[R][4], vn[R][4], zn[R][4];        // vn, zn: the next row's, where rows are walked
#pragma unroll
  for (int c = 0; c < R; ++c) {
    const int i = (c * blockDim.x + threadIdx.x) * 4;
#pragma unroll
    for (int e = 0; e < 4; ++e) { wk[c][e] = 1.f; v[c][e] = z[c][e] = vn[c][e] = zn[c][e] = 0.f; }
    if (w && i < n) load4(w + c0 + i, wk[c]);
  }
  chain_wait(y, zsrc);
  auto ask = [&](int t, float (&yv)[R][4], float (&zv)[R][4]) {
    const TY* yr = y + (size_t)t * ldy + ycol0 + c0;
    const TZ* zr = MODE ? zsrc + (size_t)t * ldz + zcol0 + c0 : nullptr;
#pragma unroll
    for (int c = 0; c < R; ++c) {
      const int i = (c * blockDim.x + threadIdx.x) * 4;
      if (i < n) {
        load4(yr + i, yv[c]);
        if (MODE) load4(zr + i, zv[c]);
      }
    }
  };
  auto norm_row = [&](int t) {
    float ss = 0.f;
#pragma unroll
    for (int c = 0; c < R; ++c)
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        if (MODE) {
          const float sg = 1.f / (1.f + expf(-z[c][e]));
          if (MODE == 1) v[c][e] *= z[c][e] * sg;
          else z[c][e] = MODE == 3 ? sg : z[c][e] * sg;
        }
        ss += v[c][e] * v[c][e];
      }
    const float inv = rsqrtf(block_sum(ss, red) / (float)n + eps);
#pragma unroll
    for (int c = 0; c < R; ++c) {
      const int i = (c * blockDim.x + threadIdx.x) * 4;
      if (i >= n) continue;
      float o[4];
#pragma unroll
      for (int e = 0; e < 4; ++e) o[e] = v[c][e] * inv * wk[c][e] * (MODE >= 2 ? z[c][e] : 1.f);
      store4(out + (size_t)t * ldo + c0 + i, o);
    }
  };
  if constexpr (WALK) {
    ask(blockIdx.x, vn, zn);
    for (int t = blockIdx.x; t < rows; t += gridDim.x) {
#pragma unroll
      for (int c = 0; c < R; ++c)
#pragma unroll
        for (int e = 0; e < 4; ++e) { v[c][e] = vn[c][e]; z[c][e] = zn[c][e]; }
      if (t + (int)gridDim.x < rows) ask(t + gridDim.x, vn, zn);
      norm_row(t);
    }
  } else {
    ask(blockIdx.x, v, z);
    norm_row(blockIdx.x);
  }
}
// Whether rows of `n` numbers at `p` (first column `col0`, `ld` apart, `el` bytes a number) can be moved four at a time.
static inline bool runs_of_four(const void* p, size_t el, long ld, long col0) {
  return ld % 4 == 0 && col0 % 4 == 0 && (uintptr_t)p % (4 * el) == 0;
}
// 0: not in the wide form
template <typename TY, typename TZ, typename T, int MODE>
static int part_norm_vec(const void* y, int ldy, int ycol0, const void* z, int ldz, int zcol0, const float* w, float eps,
                         void* out, int ldo, int R, int n, int parts, cudaStream_t stream) {
  if (n % 4 || n > 8192 || parts > 65535 || !runs_of_four(y, sizeof(TY), ldy, ycol0) || !runs_of_four(out, sizeof(T), ldo, 0) ||
      (MODE && !runs_of_four(z, sizeof(TZ), ldz, zcol0)) || (uintptr_t)w % 16)
    return 0;
  const int units = n / 4, runs = units <= 512 ? 1 : (units <= 1024 ? 2 : 4);
  const int th = ((units + runs - 1) / runs + 31) / 32 * 32;
#define NF_PN(RR, WALK, CTAS)                                                                                              \
  launch_chained(part_norm_vec_kernel<TY, TZ, T, RR, MODE, WALK>, dim3(CTAS, parts), dim3(th), 0, stream, (const TY*)y, ldy, ycol0, \
                 (const TZ*)z, ldz, zcol0, w, eps, (T*)out, ldo, n, R)
  // Rows are walked where a row is a thread's one run of four and has no gate beside it: wider ones take so many registers
  // for the next row that fewer CTAs fit (rows of 8,192 with a gate, 2,048 of them: 31 us, walked 62; of 3,584 17 and 22),
  // with a gate nothing is gained (rows of 2,048, 4,096 of them: 17.6 and 17.1, 512 of them 3.3 and 3.5; without 10.7 and 9.1).
  if (runs == 1) {
    if (MODE == 0 && parts == 1 && 2 * row_ctas(R, th) <= R) NF_PN(1, MODE == 0, row_ctas(R, th)); else NF_PN(1, false, R);
  } else if (runs == 2) {
    NF_PN(2, false, R);
  } else {
    NF_PN(4, false, R);
  }
#undef NF_PN
  return 1;
}

// out[t, 0:n] = x[t, col0:col0+n] * rsqrt(mean(x^2) + eps) * w   (w may be null: weight 1)
template <typename T>
__global__ void rms_norm_slice_kernel(const T* __restrict__ x, int ldx, int col0, int n,
                                      const float* __restrict__ w, float eps, T* __restrict__ out, int ldo) {
  __shared__ float red[33];
  const int t = blockIdx.x;
  chain_release_if_small();
  chain_wait(x);
  const T* xr = x + (size_t)t * ldx + col0;
  float ss = 0.f;
  for (int i = threadIdx.x; i < n; i += blockDim.x) {
    const float v = to_float(xr[i]);
    ss += v * v;
  }
  const float inv = rsqrtf(block_sum(ss, red) / (float)n + eps);
  T* o = out + (size_t)t * ldo;
  for (int i = threadIdx.x; i < n; i += blockDim.x)
    o[i] = from_float<T>(to_float(xr[i]) * inv * (w ? w[i] : 1.f));
}

// g = y * silu(z); each of `parts` equal parts of a row over its own root mean square; times w.
// y float32 [T, inner]; z = zsrc[t, zcol0 + i]; out [T, inner].
template <typename T>
__global__ void gated_group_rmsnorm_kernel(const float* __restrict__ y, const T* __restrict__ zsrc, int ldz,
                                           int zcol0, const float* __restrict__ w, float eps,
                                           T* __restrict__ out, int inner, int parts) {
  extern __shared__ float row[];      // [inner / parts]
  __shared__ float red[33];
  const int t = blockIdx.x, part = blockIdx.y;
  const int n = inner / parts, c0 = part * n;
  chain_release_if_small();
  chain_wait(y, zsrc);
  const float* yr = y + (size_t)t * inner + c0;
  const T* zr = zsrc + (size_t)t * ldz + zcol0 + c0;
  float ss = 0.f;
  for (int i = threadIdx.x; i < n; i += blockDim.x) {
    const float z = to_float(zr[i]);
    const float g = yr[i] * (z / (1.f + expf(-z)));
    row[i] = g;
    ss += g * g;
  }
  const float inv = rsqrtf(block_sum(ss, red) / (float)n + eps);
  T* o = out + (size_t)t * inner + c0;
  for (int i = threadIdx.x; i < n; i += blockDim.x) o[i] = from_float<T>(row[i] * inv * w[c0 + i]);
}

__global__ void add_row_vector_kernel(float* __restrict__ h, const float* __restrict__ vec, int hidden) {
  chain_wait(h);
  float* hr = h + (size_t)blockIdx.x * hidden;
  for (int i = threadIdx.x; i < hidden; i += blockDim.x) hr[i] += vec[i];
}

// out[t, hd * n + i] = v[hd, t, i] * sigmoid(g[t, gcol0 + hd * n + i]):  v is laid out head by head
// ([heads, T, n], what a batched product over heads leaves), out token by token.
// Runs of four (n a multiple of 4, rows aligned), one a thread: see heads_sigmoid_gate_kernel.
template <typename T>
__global__ void __launch_bounds__(256)
heads_sigmoid_gate_vec_kernel(const T* __restrict__ v, const T* __restrict__ g, int ldg, int gcol0, T* __restrict__ out, int rows,
                              int heads, int n, int per_head) {
  const int t = blockIdx.x, c = (blockIdx.y * 256 + threadIdx.x) * 4;
  chain_release_if_small();
  chain_wait(v, g);
  if (c >= heads * n) return;
  const int hd = c / n, i = c - hd * n;
  float x[4], gv[4];
  load4(v + ((size_t)hd * rows + t) * n + i, x);
  if (per_head) gv[0] = gv[1] = gv[2] = gv[3] = to_float(g[(size_t)t * ldg + gcol0 + hd]);
  else load4(g + (size_t)t * ldg + gcol0 + c, gv);
#pragma unroll
  for (int e = 0; e < 4; ++e) x[e] *= 1.f / (1.f + expf(-gv[e]));
  store4(out + (size_t)t * heads * n + c, x);
}

template <typename T>
__global__ void heads_sigmoid_gate_kernel(const T* __restrict__ v, const T* __restrict__ g, int ldg, int gcol0,
                                          T* __restrict__ out, int rows, int heads, int n, int per_head) {
  const int t = blockIdx.x;
  chain_wait(v, g);
  const int width = heads * n;
  for (int c = threadIdx.x; c < width; c += blockDim.x) {
    const int hd = c / n, i = c - hd * n;
    const float gv = to_float(g[(size_t)t * ldg + gcol0 + (per_head ? hd : c)]);
    const float vv = to_float(v[((size_t)hd * rows + t) * n + i]);
    out[(size_t)t * width + c] = from_float<T>(vv * (1.f / (1.f + expf(-gv))));
  }
}

// out[p] = scale[order[p]] * x[order[p] / div]: the tokens in the experts' order, each times the
// weight of its (token, choice) pair.  VEC: 16 bytes a thread and step (rows are 16-byte aligned).
template <typename T, bool VEC>
__global__ void scale_gather_rows_kernel(const T* __restrict__ x, const int* __restrict__ order, int div,
                                         const float* __restrict__ scale, T* __restrict__ out, int hidden,
                                         int n_pairs) {
  constexpr int VE = 16 / (int)sizeof(T);
  const int p = blockIdx.x;
  chain_wait(x, order, scale);
  const int pair = order[p];
  T* o = out + (size_t)p * hidden;
  const bool bad = pair < 0 || pair >= n_pairs;
  const float s = bad ? 0.f : scale[pair];
  const T* xr = x + (size_t)(bad ? 0 : pair / div) * hidden;
  if (VEC) {
    for (int i = threadIdx.x * VE; i < hidden; i += blockDim.x * VE) {
      float v[8];
      if (sizeof(T) == 2) load8(reinterpret_cast<const __nv_bfloat16*>(xr) + i, v);
      else load4(reinterpret_cast<const float*>(xr) + i, v);
#pragma unroll
      for (int e = 0; e < VE; ++e) v[e] = bad ? 0.f : s * v[e];
      if (sizeof(T) == 2) {
        store4(reinterpret_cast<__nv_bfloat16*>(o) + i, v);
        store4(reinterpret_cast<__nv_bfloat16*>(o) + i + 4, v + 4);
      } else {
        store4(reinterpret_cast<float*>(o) + i, v);
      }
    }
  } else {
    for (int i = threadIdx.x; i < hidden; i += blockDim.x) o[i] = from_float<T>(bad ? 0.f : s * to_float(xr[i]));
  }
}

}  // namespace nf

using namespace nf;

extern "C" int nf_add_layernorm(float* h, const void* delta, const int* rows, const float* w, float eps, void* out,
                                int R, int hidden, int dtype, const void* y, const int* inv, const float* wts, int k,
                                cudaStream_t stream) {
  if (R == 0) return 0;
  NF_REQUIRE(R > 0 && hidden > 0, "add_layernorm: bad sizes R=%d hidden=%d", R, hidden);
  const size_t smem = (size_t)hidden * sizeof(float);
  NF_REQUIRE(smem <= 160 * 1024, "add_layernorm: a row of %d does not fit shared memory", hidden);
  const int threads = hidden >= 2048 ? 512 : 256;
  const int runs = (hidden / 4 + threads - 1) / threads;
#define NF_LN_R(T, RR, WALK)                                                                                            \
  launch_chained(add_layernorm_regs_kernel<T, RR, WALK>, dim3(WALK ? row_ctas(R, threads) : R), dim3(threads), 0, stream, h, \
                 (const T*)delta, w, eps, (T*)out, hidden, R)
  // (rows of more than a run a thread take so many registers for the next one that fewer CTAs fit: they are not walked)
#define NF_LN_REGS(T)                                                                                                   \
  do {                                                                                                                  \
    if (runs <= 1) { if (2 * row_ctas(R, threads) <= R) NF_LN_R(T, 1, true); else NF_LN_R(T, 1, false); }                    \
    else if (runs <= 2) NF_LN_R(T, 2, false);                                                                           \
    else NF_LN_R(T, 4, false);                                                                                          \
  } while (0)
#define NF_LN(T, G, V)                                                                                      \
  do {                                                                                                      \
    if (smem > 48 * 1024)                                                                                   \
      cudaFuncSetAttribute(add_layernorm_kernel<T, G, V>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem); \
    launch_chained(add_layernorm_kernel<T, G, V>, dim3(R), dim3(threads), smem, stream, h, (const T*)delta, rows, w, \
                   eps, (T*)out, hidden, (const T*)y, inv, wts, k);                                         \
  } while (0)
#define NF_LN_V(T, G) do { if (vec) NF_LN(T, G, true); else NF_LN(T, G, false); } while (0)
  const size_t tsize = dtype == kF32 ? 4 : 2;
  const bool vec = hidden % 4 == 0 && (uintptr_t)h % 16 == 0 && (uintptr_t)w % 16 == 0 && (uintptr_t)out % (4 * tsize) == 0 &&
                   (!delta || (uintptr_t)delta % (4 * tsize) == 0) && (!y || (uintptr_t)y % (4 * tsize) == 0);
  if (vec && !rows && !y && runs <= 4) {
    if (dtype == kF32) NF_LN_REGS(float); else NF_LN_REGS(__nv_bfloat16);
  } else if (dtype == kF32) {
    if (rows) NF_LN_V(float, true); else NF_LN_V(float, false);
  } else {
    if (rows) NF_LN_V(__nv_bfloat16, true); else NF_LN_V(__nv_bfloat16, false);
  }
#undef NF_LN_V
#undef NF_LN_REGS
#undef NF_LN_R
#undef NF_LN
  return check_launch("add_layernorm");
}

// h float32 [T, hidden] (updated in place unless `rows`), d1 / d2 [T, hidden] in `dtype` or null, out [R, hidden].
extern "C" int nf_add_group_rmsnorm(float* h, const void* d1, const void* d2, const int* rows, const float* w, float eps,
                                    int groups, void* out, int R, int hidden, int dtype, cudaStream_t stream) {
  if (R == 0) return 0;
  NF_REQUIRE(R > 0 && hidden > 0 && w && groups >= 1 && hidden % groups == 0, "add_group_rmsnorm: %d groups of a row of %d", groups, hidden);
  const size_t el = dtype == kF32 ? 4 : 2;
  const bool vec = (hidden / groups) % 4 == 0 && (uintptr_t)h % 16 == 0 && (uintptr_t)w % 16 == 0 &&
                   (uintptr_t)out % (4 * el) == 0 && (uintptr_t)d1 % (4 * el) == 0 && (uintptr_t)d2 % (4 * el) == 0;
  int th = 64;
  while (th < (vec ? hidden / 4 : hidden) && th < 256) th <<= 1;
  const int nwarp = th / 32, wpg = nwarp > groups ? nwarp / groups : 1;
  const size_t smem = ((size_t)hidden + (size_t)groups * (wpg + 1)) * sizeof(float);
  NF_REQUIRE(smem <= 200 * 1024, "add_group_rmsnorm: a row of %d does not fit shared memory", hidden);
#define NF_GN(TT, GA, VE)                                                                                             \
  do {                                                                                                                \
    if (smem > 48 * 1024) cudaFuncSetAttribute(add_group_rmsnorm_kernel<TT, GA, VE>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem); \
    launch_chained(add_group_rmsnorm_kernel<TT, GA, VE>, dim3(R), dim3(th), smem, stream, h, (const TT*)d1,           \
                   (const TT*)d2, rows, w, eps, groups, (TT*)out, hidden);                                            \
  } while (0)
#define NF_GN2(TT)                                                                                                    \
  do {                                                                                                                \
    if (rows) { if (vec) NF_GN(TT, true, true); else NF_GN(TT, true, false); }                                        \
    else { if (vec) NF_GN(TT, false, true); else NF_GN(TT, false, false); }                                           \
  } while (0)
  if (dtype == kF32) NF_GN2(float); else NF_GN2(__nv_bfloat16);
#undef NF_GN2
#undef NF_GN
  return check_launch("add_group_rmsnorm");
}

extern "C" int nf_rms_norm_slice(const void* x, int ldx, int col0, int n, const float* w, float eps, void* out,
                                 int ldo, int R, int dtype, cudaStream_t stream) {
  if (R == 0) return 0;
  NF_REQUIRE(R > 0 && n > 0 && col0 >= 0 && col0 + n <= ldx && ldo >= n, "rms_norm_slice: bad sizes");
  if (dtype == kF32 ? part_norm_vec<float, float, float, 0>(x, ldx, col0, nullptr, 0, 0, w, eps, out, ldo, R, n, 1, stream)
                    : part_norm_vec<__nv_bfloat16, float, __nv_bfloat16, 0>(x, ldx, col0, nullptr, 0, 0, w, eps, out, ldo, R, n, 1, stream))
    return check_launch("rms_norm_slice");
  if (dtype == kF32)
    launch_chained(rms_norm_slice_kernel<float>, dim3(R), dim3(128), 0, stream, (const float*)x, ldx, col0, n, w, eps, (float*)out, ldo);
  else
    launch_chained(rms_norm_slice_kernel<__nv_bfloat16>, dim3(R), dim3(128), 0, stream, (const __nv_bfloat16*)x, ldx, col0, n, w, eps, (__nv_bfloat16*)out, ldo);
  return check_launch("rms_norm_slice");
}

extern "C" int nf_gated_group_rmsnorm(const float* y, const void* z, int ldz, int zcol0, const float* w, float eps,
                                      void* out, int R, int inner, int parts, int dtype, cudaStream_t stream) {
  if (R == 0) return 0;
  NF_REQUIRE(R > 0 && inner > 0 && parts > 0 && inner % parts == 0, "gated_group_rmsnorm: %d does not split into %d parts", inner, parts);
  if (dtype == kF32 ? part_norm_vec<float, float, float, 1>(y, inner, 0, z, ldz, zcol0, w, eps, out, inner, R, inner / parts, parts, stream)
                    : part_norm_vec<float, __nv_bfloat16, __nv_bfloat16, 1>(y, inner, 0, z, ldz, zcol0, w, eps, out, inner, R, inner / parts, parts, stream))
    return check_launch("gated_group_rmsnorm");
  const size_t smem = (size_t)(inner / parts) * sizeof(float);
  NF_REQUIRE(smem <= 160 * 1024, "gated_group_rmsnorm: a part of %d does not fit shared memory", inner / parts);
#define NF_GN(T)                                                                                               \
  do {                                                                                                         \
    if (smem > 48 * 1024)                                                                                      \
      cudaFuncSetAttribute(gated_group_rmsnorm_kernel<T>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem); \
    launch_chained(gated_group_rmsnorm_kernel<T>, dim3(R, parts), dim3(256), smem, stream, y, (const T*)z, ldz, zcol0, \
                   w, eps, (T*)out, inner, parts);                                                             \
  } while (0)
  if (dtype == kF32) NF_GN(float); else NF_GN(__nv_bfloat16);
#undef NF_GN
  return check_launch("gated_group_rmsnorm");
}

extern "C" int nf_add_row_vector(float* h, const float* vec, int R, int hidden, cudaStream_t stream) {
  if (R == 0) return 0;
  launch_chained(add_row_vector_kernel, dim3(R), dim3(256), 0, stream, h, vec, hidden);
  return check_launch("add_row_vector");
}

// per_head != 0: the gate has one logit a head (column gcol0 + head) instead of one an element
extern "C" int nf_heads_sigmoid_gate(const void* v, const void* g, int ldg, int gcol0, void* out, int R, int heads,
                                     int n, int per_head, int dtype, cudaStream_t stream) {
  if (R == 0) return 0;
  NF_REQUIRE(heads > 0 && n > 0 && gcol0 >= 0 && gcol0 + heads * (per_head ? 1 : n) <= ldg, "heads_sigmoid_gate: bad sizes");
  const size_t el = dtype == kF32 ? 4 : 2;
  if (n % 4 == 0 && runs_of_four(v, el, 0, 0) && runs_of_four(out, el, 0, 0) && (per_head || runs_of_four(g, el, ldg, gcol0))) {
    const dim3 grid(R, (heads * n / 4 + 255) / 256);
    if (dtype == kF32) launch_chained(heads_sigmoid_gate_vec_kernel<float>, grid, dim3(256), 0, stream, (const float*)v, (const float*)g, ldg, gcol0, (float*)out, R, heads, n, per_head);
    else launch_chained(heads_sigmoid_gate_vec_kernel<__nv_bfloat16>, grid, dim3(256), 0, stream, (const __nv_bfloat16*)v, (const __nv_bfloat16*)g, ldg, gcol0, (__nv_bfloat16*)out, R, heads, n, per_head);
    return check_launch("heads_sigmoid_gate");
  }
  if (dtype == kF32)
    launch_chained(heads_sigmoid_gate_kernel<float>, dim3(R), dim3(256), 0, stream, (const float*)v, (const float*)g, ldg, gcol0, (float*)out, R, heads, n, per_head);
  else
    launch_chained(heads_sigmoid_gate_kernel<__nv_bfloat16>, dim3(R), dim3(256), 0, stream, (const __nv_bfloat16*)v, (const __nv_bfloat16*)g, ldg, gcol0, (__nv_bfloat16*)out, R, heads, n, per_head);
  return check_launch("heads_sigmoid_gate");
}

extern "C" int nf_scale_gather_rows(const void* x, const int* order, int div, const float* scale, void* out,
                                    int n_rows, int hidden, int dtype, cudaStream_t stream) {
  if (n_rows == 0) return 0;
  NF_REQUIRE(div > 0 && hidden > 0, "scale_gather_rows: bad sizes");
  const int threads = hidden >= 2048 ? 256 : 128;
  if (dtype == kF32) {
    if (hidden % 4 == 0) launch_chained(scale_gather_rows_kernel<float, true>, dim3(n_rows), dim3(threads), 0, stream, (const float*)x, order, div, scale, (float*)out, hidden, n_rows);
    else launch_chained(scale_gather_rows_kernel<float, false>, dim3(n_rows), dim3(256), 0, stream, (const float*)x, order, div, scale, (float*)out, hidden, n_rows);
  } else {
    if (hidden % 8 == 0) launch_chained(scale_gather_rows_kernel<__nv_bfloat16, true>, dim3(n_rows), dim3(threads), 0, stream, (const __nv_bfloat16*)x, order, div, scale, (__nv_bfloat16*)out, hidden, n_rows);
    else launch_chained(scale_gather_rows_kernel<__nv_bfloat16, false>, dim3(n_rows), dim3(256), 0, stream, (const __nv_bfloat16*)x, order, div, scale, (__nv_bfloat16*)out, hidden, n_rows);
  }
  return check_launch("scale_gather_rows");
}

// ---------------------------------------------------------------------------------------------
// Norm on a sublayer's output: h[t] += ls * (d / rms(d)) * w with d = delta[t] (+ bias), and, if
// `out`, out[t] = h[t] in the engine's type (the next sublayer's input).  delta may be float32 or
// the engine's type; the sum, the mean of squares and the products are float32.
// ---------------------------------------------------------------------------------------------
namespace nf {

// One element of the update, in the kernels below to the last bit alike: (d / rms) * w (* scale) added to the stream.
__device__ __forceinline__ float scaled_norm_sum(float d, float inv, float w, const float* ls, float scale, float h) {
  const float t = d * inv;
  return ls ? fmaf(t * w, scale, h) : fmaf(t, w, h);
}

template <typename TD, typename TO>
__global__ void scaled_norm_add_kernel(float* __restrict__ h, const TD* __restrict__ delta,
                                       const float* __restrict__ bias, const float* __restrict__ w,
                                       const float* __restrict__ ls, float eps, TO* __restrict__ out, int hidden) {
  __shared__ float red[33];
  const int r = blockIdx.x;
  chain_release_if_small();
  chain_wait(h, delta);
  float* hr = h + (size_t)r * hidden;
  const TD* dr = delta + (size_t)r * hidden;
  float ss = 0.f;
  for (int i = threadIdx.x; i < hidden; i += blockDim.x) {
    const float d = to_float(dr[i]) + (bias ? bias[i] : 0.f);
    ss = fmaf(d, d, ss);
  }
  const float inv = rsqrtf(block_sum(ss, red) / (float)hidden + eps);
  for (int i = threadIdx.x; i < hidden; i += blockDim.x) {
    const float d = to_float(dr[i]) + (bias ? bias[i] : 0.f);
    const float v = scaled_norm_sum(d, inv, w[i], ls, ls ? ls[i] : 1.f, hr[i]);
    hr[i] = v;
    if (out) out[(size_t)r * hidden + i] = from_float<TO>(v);
  }
}

// Rows of up to R numbers a thread: the same sums in the same order, with the row in registers between the two passes, all
// its numbers asked for at once and the weights, which no kernel writes, before the wait (see part_norm_vec_kernel).
template <typename TD, typename TO, int R, bool WALK>
__global__ void __launch_bounds__(512)
scaled_norm_add_regs_kernel(float* __restrict__ h, const TD* __restrict__ delta, const float* __restrict__ bias,
                            const float* __restrict__ w, const float* __restrict__ ls, float eps, TO* __restrict__ out, int hidden,
                            int rows) {
  __shared__ float red[33];
  chain_release_if_small();
  float wk[R], lk[R], bk[R], d[R], hk[R], hn[R];      // hn: the next row's, where rows are walked
#pragma unroll
  for (int c = 0; c < R; ++c) {
    const int i = c * blockDim.x + threadIdx.x;
    wk[c] = lk[c] = 1.f;
    bk[c] = d[c] = hk[c] = hn[c] = 0.f;
    if (i < hidden) {
      wk[c] = w[i];
      if (ls) lk[c] = ls[i];
      if (bias) bk[c] = bias[i];
    }
  }
  chain_wait(h, delta);
  TD raw[R];
  auto ask = [&](int r, float (&hv)[R]) {
    const float* hr = h + (size_t)r * hidden;
    const TD* dr = delta + (size_t)r * hidden;
#pragma unroll
    for (int c = 0; c < R; ++c) {
      const int i = c * blockDim.x + threadIdx.x;
      if (i < hidden) { raw[c] = dr[i]; hv[c] = hr[i]; }
    }
  };
  auto sum_row = [&]() {
    float ss = 0.f;
#pragma unroll
    for (int c = 0; c < R; ++c)
      if (c * (int)blockDim.x + (int)threadIdx.x < hidden) {
        d[c] = to_float(raw[c]) + bk[c];
        ss = fmaf(d[c], d[c], ss);
      }
    return ss;
  };
  auto add_row = [&](int r, float ss) {
    const float inv = rsqrtf(block_sum(ss, red) / (float)hidden + eps);
#pragma unroll
    for (int c = 0; c < R; ++c) {
      const int i = c * blockDim.x + threadIdx.x;
      if (i >= hidden) continue;
      const float v = scaled_norm_sum(d[c], inv, wk[c], ls, lk[c], hk[c]);
      h[(size_t)r * hidden + i] = v;
      if (out) out[(size_t)r * hidden + i] = from_float<TO>(v);
    }
  };
  if constexpr (!WALK) {
    ask(blockIdx.x, hk);
    add_row(blockIdx.x, sum_row());
  } else if constexpr (R < 16) {
    ask(blockIdx.x, hn);
    for (int r = blockIdx.x; r < rows; r += gridDim.x) {
      const float ss = sum_row();
#pragma unroll
      for (int c = 0; c < R; ++c) hk[c] = hn[c];
      if (r + (int)gridDim.x < rows) ask(r + gridDim.x, hn);
      add_row(r, ss);
    }
  } else {                             // (no registers for a next row)
    for (int r = blockIdx.x; r < rows; r += gridDim.x) {
      ask(r, hk);
      add_row(r, sum_row());
    }
  }
}

// The same with the routed experts' pending sum as the sublayer's output:
// d = sum_j wts[t, j] * y[inv[t * k + j]] (j ascending; wts null: unit weights), rounded to T as the separate
// combine kernel rounds it, so both ways give the same bits.  The row is kept in shared memory.
template <typename T, typename TO>
__global__ void routed_scaled_norm_add_kernel(float* __restrict__ h, const T* __restrict__ y, const int* __restrict__ inv,
                                              const float* __restrict__ wts, int k, const float* __restrict__ w,
                                              const float* __restrict__ ls, float eps, TO* __restrict__ out, int hidden) {
  extern __shared__ float row[];      // [hidden]
  __shared__ float red[33];
  const int r = blockIdx.x;
  chain_release_if_small();
  chain_wait(h, y, inv, wts);
  float ss = 0.f;
  for (int i = threadIdx.x; i < hidden; i += blockDim.x) {
    float acc = 0.f;
    for (int j = 0; j < k; ++j) {
      const int p = inv[r * k + j];
      acc += (wts ? wts[r * k + j] : 1.f) * to_float(y[(size_t)p * hidden + i]);
    }
    const float d = to_float(from_float<T>(acc));
    row[i] = d;
    ss = fmaf(d, d, ss);
  }
  const float invr = rsqrtf(block_sum(ss, red) / (float)hidden + eps);
  float* hr = h + (size_t)r * hidden;
  for (int i = threadIdx.x; i < hidden; i += blockDim.x) {
    const float v = scaled_norm_sum(row[i], invr, w[i], ls, ls ? ls[i] : 1.f, hr[i]);
    hr[i] = v;
    if (out) out[(size_t)r * hidden + i] = from_float<TO>(v);
  }
}

// out[t] = (1 / n) * sum_m (x_m[t] / rms(x_m[t])) * w_m: the mean of several mixers' outputs, each
// first over its own root mean square and times its own weight.  out is float32.
struct NormedInputs {
  const void* x[4];
  const float* w[4];
  int n;
};

template <typename T>
__global__ void mean_of_rmsnorms_kernel(NormedInputs in, float eps, float* __restrict__ out, int hidden) {
  __shared__ float red[33];
  const int r = blockIdx.x;
  chain_release_if_small();
  chain_wait();
  float inv[4];
  for (int m = 0; m < in.n; ++m) {
    const T* xr = reinterpret_cast<const T*>(in.x[m]) + (size_t)r * hidden;
    float ss = 0.f;
    for (int i = threadIdx.x; i < hidden; i += blockDim.x) {
      const float v = to_float(xr[i]);
      ss += v * v;
    }
    inv[m] = rsqrtf(block_sum(ss, red) / (float)hidden + eps);
  }
  const float share = 1.f / (float)in.n;
  for (int i = threadIdx.x; i < hidden; i += blockDim.x) {
    float s = 0.f;
    for (int m = 0; m < in.n; ++m)
      s += to_float(reinterpret_cast<const T*>(in.x[m])[(size_t)r * hidden + i]) * inv[m] * in.w[m][i];
    out[(size_t)r * hidden + i] = s * share;
  }
}

// The wide form for two inputs: both rows in registers, their sums of squares meet in one pass over the block.
template <typename T, int R>
__global__ void __launch_bounds__(512)
mean_of_two_rmsnorms_vec_kernel(const T* __restrict__ a, const T* __restrict__ b, const float* __restrict__ wa,
                                const float* __restrict__ wb, float eps, float* __restrict__ out, int hidden) {
  __shared__ float2 red[17];
  const int r = blockIdx.x, warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nwarp = blockDim.x >> 5;
  chain_release_if_small();
  float wk[2][R][4], v[2][R][4];
#pragma unroll
  for (int c = 0; c < R; ++c) {
    const int i = (c * blockDim.x + threadIdx.x) * 4;
#pragma unroll
    for (int e = 0; e < 4; ++e) wk[0][c][e] = wk[1][c][e] = v[0][c][e] = v[1][c][e] = 0.f;
    if (i < hidden) { load4(wa + i, wk[0][c]); load4(wb + i, wk[1][c]); }
  }
  chain_wait(a, b);
#pragma unroll
  for (int c = 0; c < R; ++c) {
    const int i = (c * blockDim.x + threadIdx.x) * 4;
    if (i < hidden) { load4(a + (size_t)r * hidden + i, v[0][c]); load4(b + (size_t)r * hidden + i, v[1][c]); }
  }
  float s0 = 0.f, s1 = 0.f;
#pragma unroll
  for (int c = 0; c < R; ++c)
#pragma unroll
    for (int e = 0; e < 4; ++e) { s0 += v[0][c][e] * v[0][c][e]; s1 += v[1][c][e] * v[1][c][e]; }
  s0 = warp_sum(s0);
  s1 = warp_sum(s1);
  if (lane == 0) red[warp] = make_float2(s0, s1);
  __syncthreads();
  if (warp == 0) {
    const float2 x = lane < nwarp ? red[lane] : make_float2(0.f, 0.f);
    s0 = warp_sum(x.x);
    s1 = warp_sum(x.y);
    if (lane == 0) red[16] = make_float2(s0, s1);
  }
  __syncthreads();
  const float i0 = rsqrtf(red[16].x / (float)hidden + eps), i1 = rsqrtf(red[16].y / (float)hidden + eps);
#pragma unroll
  for (int c = 0; c < R; ++c) {
    const int i = (c * blockDim.x + threadIdx.x) * 4;
    if (i >= hidden) continue;
    float o[4];
#pragma unroll
    for (int e = 0; e < 4; ++e) o[e] = (v[0][c][e] * i0 * wk[0][c][e] + v[1][c][e] * i1 * wk[1][c][e]) * 0.5f;
    store4(out + (size_t)r * hidden + i, o);
  }
}

// out[t, c] = y[t, c] / rms(part of c) * w[c] * act(z[t, zcol0 + c]): an RMS norm in `parts` equal
// parts of a row (w null: no weight), then a gate.  act 0: silu, 1: sigmoid.  y is float32; z is of the
// output's type or float32 sums.
template <typename T, typename TZ = T>
__global__ void group_rmsnorm_gate_kernel(const float* __restrict__ y, const TZ* __restrict__ zsrc, int ldz, int zcol0,
                                          const float* __restrict__ w, float eps, T* __restrict__ out, int inner,
                                          int parts, int act) {
  __shared__ float red[33];
  const int t = blockIdx.x, part = blockIdx.y;
  const int n = inner / parts, c0 = part * n;
  chain_release_if_small();
  chain_wait(y, zsrc);
  const float* yr = y + (size_t)t * inner + c0;
  const TZ* zr = zsrc + (size_t)t * ldz + zcol0 + c0;
  float ss = 0.f;
  for (int i = threadIdx.x; i < n; i += blockDim.x) ss += yr[i] * yr[i];
  const float inv = rsqrtf(block_sum(ss, red) / (float)n + eps);
  T* o = out + (size_t)t * inner + c0;
  for (int i = threadIdx.x; i < n; i += blockDim.x) {
    const float z = to_float(zr[i]);
    const float sg = 1.f / (1.f + expf(-z));
    const float gate = act == 1 ? sg : z * sg;
    o[i] = from_float<T>(yr[i] * inv * (w ? w[c0 + i] : 1.f) * gate);
  }
}

static inline int norm_threads(int n) {
  int t = 32;
  while (t < n && t < 512) t <<= 1;
  return t;
}

}  // namespace nf

// delta_dtype: 0 float32, 1 bfloat16; out (may be null) has out_dtype.
extern "C" int nf_scaled_norm_add(float* h, const void* delta, int delta_dtype, const float* bias, const float* w,
                                  const float* ls, float eps, void* out, int out_dtype, int R, int hidden,
                                  cudaStream_t stream) {
  if (R == 0) return 0;
  NF_REQUIRE(R > 0 && hidden > 0 && h && delta && w, "scaled_norm_add: bad arguments R=%d hidden=%d", R, hidden);
  const dim3 grid(R), block(norm_threads(hidden));
  const int each = (hidden + (int)block.x - 1) / (int)block.x;
  // Rows are walked from two a CTA on.  (257 rows of 3,584 4.9 us, as walks of one row 5.4; 512 of 4,096, walks of one or
  // two, 9.0 and 9.6; 1,024 20.5 and 16.1; rows of 256 gain nothing: 2,048 of them 5.5 and 5.7.)
  const bool walk = hidden >= 512 && 2 * row_ctas(R, (int)block.x) <= R;
#define NF_SNV(TD, TO, RR)                                                                                                 \
  do {                                                                                                                     \
    if (walk) launch_chained(scaled_norm_add_regs_kernel<TD, TO, RR, true>, dim3(row_ctas(R, (int)block.x)), block, 0, stream, h, \
                             (const TD*)delta, bias, w, ls, eps, (TO*)out, hidden, R);                                     \
    else launch_chained(scaled_norm_add_regs_kernel<TD, TO, RR, false>, dim3(R), block, 0, stream, h, (const TD*)delta, bias, w,  \
                        ls, eps, (TO*)out, hidden, R);                                                                     \
  } while (0)
#define NF_SNA(TD, TO)                                                                                                     \
  do {                                                                                                                     \
    if (each <= 4) NF_SNV(TD, TO, 4); else if (each <= 8) NF_SNV(TD, TO, 8); else if (each <= 16) NF_SNV(TD, TO, 16);      \
    else launch_chained(scaled_norm_add_kernel<TD, TO>, grid, block, 0, stream, h, (const TD*)delta, bias, w, ls, eps, (TO*)out, hidden); \
  } while (0)
  if (delta_dtype == kF32) { if (out_dtype == kF32) NF_SNA(float, float); else NF_SNA(float, __nv_bfloat16); }
  else { if (out_dtype == kF32) NF_SNA(__nv_bfloat16, float); else NF_SNA(__nv_bfloat16, __nv_bfloat16); }
#undef NF_SNA
#undef NF_SNV
  return check_launch("scaled_norm_add");
}

// y [pairs, hidden] of `dtype`, inv int32 [R * k], wts float32 [R, k] or null; out (may be null) has out_dtype.
extern "C" int nf_routed_scaled_norm_add(float* h, const void* y, const int* inv, const float* wts, int k, int dtype,
                                         const float* w, const float* ls, float eps, void* out, int out_dtype, int R,
                                         int hidden, cudaStream_t stream) {
  if (R == 0) return 0;
  NF_REQUIRE(R > 0 && hidden > 0 && k > 0 && h && y && inv && w, "routed_scaled_norm_add: bad arguments");
  const size_t smem = (size_t)hidden * sizeof(float);
  NF_REQUIRE(smem <= 160 * 1024, "routed_scaled_norm_add: a row of %d does not fit shared memory", hidden);
  const dim3 grid(R), block(norm_threads(hidden));
#define NF_RSNA(T, TO)                                                                                              \
  do {                                                                                                              \
    if (smem > 48 * 1024)                                                                                           \
      cudaFuncSetAttribute(routed_scaled_norm_add_kernel<T, TO>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem); \
    launch_chained(routed_scaled_norm_add_kernel<T, TO>, grid, block, smem, stream, h, (const T*)y, inv, wts, k, w, ls, eps, \
                   (TO*)out, hidden);                                                                               \
  } while (0)
  if (dtype == kF32) NF_RSNA(float, float);
  else if (out_dtype == kF32) NF_RSNA(__nv_bfloat16, float);
  else NF_RSNA(__nv_bfloat16, __nv_bfloat16);
#undef NF_RSNA
  return check_launch("routed_scaled_norm_add");
}

extern "C" int nf_mean_of_rmsnorms(const void* const* xs, const float* const* ws, int n, float eps, float* out, int R,
                                   int hidden, int dtype, cudaStream_t stream) {
  if (R == 0) return 0;
  NF_REQUIRE(n >= 1 && n <= 4 && R > 0 && hidden > 0, "mean_of_rmsnorms: %d inputs (1 to 4), R=%d hidden=%d", n, R, hidden);
  NormedInputs in;
  in.n = n;
  for (int m = 0; m < 4; ++m) { in.x[m] = m < n ? xs[m] : nullptr; in.w[m] = m < n ? ws[m] : nullptr; }
  const size_t el = dtype == kF32 ? 4 : 2;
  if (n == 2 && hidden % 4 == 0 && hidden <= 4096 && runs_of_four(in.x[0], el, 0, 0) && runs_of_four(in.x[1], el, 0, 0) &&
      ((uintptr_t)in.w[0] | (uintptr_t)in.w[1] | (uintptr_t)out) % 16 == 0) {
    const int units = hidden / 4, runs = units <= 512 ? 1 : 2, th = ((units + runs - 1) / runs + 31) / 32 * 32;
#define NF_MR(TT, RR) launch_chained(mean_of_two_rmsnorms_vec_kernel<TT, RR>, dim3(R), dim3(th), 0, stream, (const TT*)in.x[0], (const TT*)in.x[1], in.w[0], in.w[1], eps, out, hidden)
    if (dtype == kF32) { if (runs == 1) NF_MR(float, 1); else NF_MR(float, 2); }
    else { if (runs == 1) NF_MR(__nv_bfloat16, 1); else NF_MR(__nv_bfloat16, 2); }
#undef NF_MR
    return check_launch("mean_of_rmsnorms");
  }
  if (dtype == kF32) launch_chained(mean_of_rmsnorms_kernel<float>, dim3(R), dim3(norm_threads(hidden)), 0, stream, in, eps, out, hidden);
  else launch_chained(mean_of_rmsnorms_kernel<__nv_bfloat16>, dim3(R), dim3(norm_threads(hidden)), 0, stream, in, eps, out, hidden);
  return check_launch("mean_of_rmsnorms");
}

// z_dtype: the gate's type, the output's or float32.
extern "C" int nf_group_rmsnorm_gate(const float* y, const void* z, int ldz, int zcol0, const float* w, float eps,
                                     void* out, int R, int inner, int parts, int act, int dtype, int z_dtype,
                                     cudaStream_t stream) {
  if (R == 0) return 0;
  NF_REQUIRE(R > 0 && inner > 0 && parts > 0 && inner % parts == 0 && parts <= 65535,
             "group_rmsnorm_gate: %d does not split into %d parts", inner, parts);
  NF_REQUIRE(act == 0 || act == 1, "group_rmsnorm_gate: gate %d (0 silu, 1 sigmoid)", act);
  NF_REQUIRE(z_dtype == dtype || z_dtype == kF32, "group_rmsnorm_gate: the gate is of the output's type or float32");
  const int n = inner / parts;
#define NF_GV(TZ, T) (act == 1 ? part_norm_vec<float, TZ, T, 3>(y, inner, 0, z, ldz, zcol0, w, eps, out, inner, R, n, parts, stream) \
                               : part_norm_vec<float, TZ, T, 2>(y, inner, 0, z, ldz, zcol0, w, eps, out, inner, R, n, parts, stream))
  if (dtype == kF32 ? NF_GV(float, float) : (z_dtype == kF32 ? NF_GV(float, __nv_bfloat16) : NF_GV(__nv_bfloat16, __nv_bfloat16)))
    return check_launch("group_rmsnorm_gate");
#undef NF_GV
  const dim3 grid(R, parts), block(norm_threads(n));
  if (dtype == kF32) launch_chained(group_rmsnorm_gate_kernel<float>, grid, block, 0, stream, y, (const float*)z, ldz, zcol0, w, eps, (float*)out, inner, parts, act);
  else if (z_dtype == kF32) launch_chained(group_rmsnorm_gate_kernel<__nv_bfloat16, float>, grid, block, 0, stream, y, (const float*)z, ldz, zcol0, w, eps, (__nv_bfloat16*)out, inner, parts, act);
  else launch_chained(group_rmsnorm_gate_kernel<__nv_bfloat16>, grid, block, 0, stream, y, (const __nv_bfloat16*)z, ldz, zcol0, w, eps, (__nv_bfloat16*)out, inner, parts, act);
  return check_launch("group_rmsnorm_gate");
}
