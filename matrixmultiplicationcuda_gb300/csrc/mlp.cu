// The learned cost model: a small fp32 MLP (structure features -> predicted
// log time of every tuner configuration), with its training kernels.
//
// Network: x -> (x - mu) / sigma -> [Linear -> GELU] x layers -> Linear; the
// outputs are ln(time in microseconds), one per tuner configuration.
// Parameters live in one flat fp32 array:
//   mu[in], sigma[in]                      (input normalisation, not trained)
//   W0[hidden x in], b0[hidden]            (row-major: W[o * fan_in + i])
//   W1..W{layers-1}[hidden x hidden], b
//   W_out[out x hidden], b_out[out]
// GELU is the exact form 0.5 x (1 + erf(x / sqrt 2)).
//
// Training minimises the masked mean squared error over (sample, config)
// pairs with mask 1: loss = sum(mask (y - t)^2) / sum(mask). The backward pass
// either runs fused (k_mlp_fused: a CTA takes tiles of 8 samples through all
// layers and back with the weights in shared memory, then k_mlp_reduce adds the
// CTAs' gradients in a fixed order) or, for networks whose weights do not fit
// in shared memory, layer by layer with every pre-activation and activation in
// a workspace and the weight gradients reduced over the batch inside one CTA
// per output unit. Both give the same gradient on every run. Adam updates only
// the trained range.
#include <algorithm>
#include <cmath>
#include <cstdio>
#include <cstring>
#include <vector>
#include "internal.h"
#include "ptx.cuh"

namespace spmm {
namespace {

constexpr int kFusedRows = 8;             // samples per tile of the fused path
constexpr int kFusedMaxCtas = 128;
constexpr int kFusedThreads = 256;
constexpr long long kFusedSmemMax = 200 * 1024;

// Offsets of the fused path, from a few numbers: a table of layers among the
// kernel's parameters cost a constant-cache miss per layer, 12,000 cycles
// before the first layer ran.
struct FusedLayer {
  int I, O, ld;        // fan-in, fan-out, row length of W and of the layer's input
  int w, b, act;       // W, bias and the tile's input in shared memory (floats)
  int gw, gpart;       // W in the parameter array and in a CTA's gradient
};
struct FusedShape {
  int in, hidden, layers, out, ld0, ldh;   // ld0, ldh: row length for a fan-in of `in` and of `hidden`
  __host__ __device__ static int up4(int x) { return (x + 3) & ~3; }
  __host__ __device__ FusedLayer layer(int l) const {
    FusedLayer f;
    f.I = l == 0 ? in : hidden;
    f.O = l == layers ? out : hidden;
    f.ld = l == 0 ? ld0 : ldh;
    const int before = l == 0 ? 0 : l - 1;   // whole hidden layers before this one, after the first
    f.w = up4(2 * in) + (l == 0 ? 0 : (hidden + kFusedRows) * ld0 + up4(hidden)) +
          before * ((hidden + kFusedRows) * ldh + up4(hidden));
    f.b = f.w + f.O * f.ld;
    f.act = f.b + up4(f.O);
    f.gw = 2 * in + (l == 0 ? 0 : hidden * (in + 1)) + before * hidden * (hidden + 1);
    f.gpart = (l == 0 ? 0 : up4(hidden) * (up4(in) + 1)) + before * up4(hidden) * (up4(hidden) + 1);
    return f;
  }
  __host__ __device__ int end() const {   // past the last layer's input
    const FusedLayer f = layer(layers);
    return f.act + kFusedRows * f.ld;
  }
  // GELU' of hidden layer l's outputs (the input of layer l + 1), the targets
  // and the mask of the tile, the two dZ tiles
  __host__ __device__ int gp(int l) const { return end() + (l - 1) * kFusedRows * hidden; }
  __host__ __device__ int tgt() const { return gp(layers + 1); }
  __host__ __device__ int dz() const { return up4(tgt() + 2 * kFusedRows * out); }
  __host__ __device__ int ld_dz() const { return up4(hidden > out ? hidden : out); }
  __host__ __device__ int smem_floats() const { return dz() + 2 * kFusedRows * ld_dz(); }
  __host__ __device__ int part_floats() const {
    const FusedLayer f = layer(layers);
    return f.gpart + up4(f.O) * (up4(f.I) + 1);
  }
};

struct Layout {
  int in, hidden, layers, out;
  long long norm_floats() const { return 2LL * in; }
  int fan_in(int l) const { return l == 0 ? in : hidden; }
  int fan_out(int l) const { return l == layers ? out : hidden; }
  long long w_off(int l) const {
    long long o = norm_floats();
    for (int k = 0; k < l; ++k) o += (long long)fan_out(k) * fan_in(k) + fan_out(k);
    return o;
  }
  long long b_off(int l) const { return w_off(l) + (long long)fan_out(l) * fan_in(l); }
  long long params() const { return w_off(layers + 1); }
  // workspace of the layer-by-layer path: Xn[B x in], per hidden layer
  // Z[B x hidden] and A[B x hidden], Y[B x out], two gradient buffers
  // [B x max(hidden, out)]
  long long layer_ws(int batch) const {
    const int wmax = hidden > out ? hidden : out;
    return (long long)batch * (in + 2LL * hidden * layers + out + 2LL * wmax);
  }
  FusedShape fused_shape() const {
    // row lengths are multiples of 4 floats whose quarter is odd, so that eight
    // lanes reading 16 bytes of eight rows touch all banks
    auto row = [](int n) {
      const int q = FusedShape::up4(n);
      return (q & 4) ? q : q + 4;
    };
    return FusedShape{in, hidden, layers, out, row(in), row(hidden)};
  }
  bool fused() const { return (fused_shape().smem_floats() + 64) * 4LL <= kFusedSmemMax; }
  int fused_ctas(int batch) const {
    const int tiles = (batch + kFusedRows - 1) / kFusedRows;
    return tiles < kFusedMaxCtas ? tiles : kFusedMaxCtas;
  }
  // {loss sum, mask sum} per CTA in double, then the gradients per CTA
  long long fused_ws(int batch) const { return fused_ctas(batch) * (4LL + fused_shape().part_floats()); }
  long long ws(int batch) const {
    const long long a = layer_ws(batch), b = fused() ? fused_ws(batch) : 0;
    return a > b ? a : b;
  }
};

bool valid(const spmm_mlp_shape* s) {
  // fan-ins up to 128 keep a 64-row slice of a layer's input within 32 KB of shared memory
  return s && s->in > 0 && s->hidden > 0 && s->layers > 0 && s->out > 0 && s->in <= 128 && s->hidden <= 128 &&
         s->out <= 1024 && s->layers <= 16;
}
Layout layout(const spmm_mlp_shape* s) { return Layout{s->in, s->hidden, s->layers, s->out}; }

__device__ __forceinline__ float gelu(float x) { return 0.5f * x * (1.f + erff(x * 0.70710678118654752f)); }
__device__ __forceinline__ float gelu_grad(float x) {
  // d/dx [x Phi(x)] = Phi(x) + x phi(x)
  return 0.5f * (1.f + erff(x * 0.70710678118654752f)) + x * 0.39894228040143268f * expf(-0.5f * x * x);
}

__global__ void k_normalize(const float* __restrict__ X, const float* __restrict__ mu,
                            const float* __restrict__ sigma, int batch, int in, float* __restrict__ Xn) {
  const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= (long long)batch * in) return;
  const int f = (int)(i % in);
  Xn[i] = (X[i] - mu[f]) / sigma[f];
}

// Z[b][o] = sum_i X[b][i] W[o][i] + bias[o]; A = GELU(Z) when A != NULL.
// One thread per (b, o); the CTA's 64-row slice of X is staged in shared memory.
__global__ void k_dense(const float* __restrict__ X, const float* __restrict__ W, const float* __restrict__ bias,
                        int batch, int I, int O, float* __restrict__ Z, float* __restrict__ A) {
  extern __shared__ float sx[];   // [rows x I]
  constexpr int rows = 64;
  const int b0 = blockIdx.x * rows;
  for (int t = threadIdx.x; t < rows * I; t += blockDim.x) {
    const int r = t / I, i = t % I;
    sx[t] = (b0 + r < batch) ? X[(long long)(b0 + r) * I + i] : 0.f;
  }
  __syncthreads();
  for (int t = threadIdx.x; t < rows * O; t += blockDim.x) {
    const int r = t / O, o = t % O;
    if (b0 + r >= batch) continue;
    const float* w = W + (long long)o * I;
    const float* x = sx + r * I;
    float acc = bias[o];
    for (int i = 0; i < I; ++i) acc = fmaf(x[i], __ldg(w + i), acc);
    Z[(long long)(b0 + r) * O + o] = acc;
    if (A) A[(long long)(b0 + r) * O + o] = gelu(acc);
  }
}

// Masked MSE: loss = sum(m (y - t)^2) / sum(m); dY = 2 m (y - t) / sum(m).
// One CTA (the batch is small); sums in double for a stable loss value.
__global__ void k_mse(const float* __restrict__ Y, const float* __restrict__ T, const float* __restrict__ M,
                      long long n, float* __restrict__ dY, float* __restrict__ loss) {
  __shared__ double s_sum[1024], s_cnt[1024];
  double sum = 0, cnt = 0;
  for (long long i = threadIdx.x; i < n; i += blockDim.x) {
    const float m = M[i];
    if (m != 0.f) {
      const double d = (double)Y[i] - (double)T[i];
      sum += m * d * d;
      cnt += m;
    }
  }
  s_sum[threadIdx.x] = sum;
  s_cnt[threadIdx.x] = cnt;
  __syncthreads();
  for (int w = blockDim.x / 2; w > 0; w >>= 1) {
    if ((int)threadIdx.x < w) {
      s_sum[threadIdx.x] += s_sum[threadIdx.x + w];
      s_cnt[threadIdx.x] += s_cnt[threadIdx.x + w];
    }
    __syncthreads();
  }
  const double total = s_cnt[0] > 0 ? s_cnt[0] : 1.0;
  if (threadIdx.x == 0 && loss) *loss = (float)(s_sum[0] / total);
  const float scale = (float)(2.0 / total);
  for (long long i = threadIdx.x; i < n; i += blockDim.x) {
    const float m = M[i];
    dY[i] = m != 0.f ? scale * m * (Y[i] - T[i]) : 0.f;
  }
}

// dW[o][i] = sum_b dZ[b][o] X[b][i]; db[o] = sum_b dZ[b][o]. One CTA per o;
// thread t takes input i = t % I and the batch rows b = t / I (mod slices).
__global__ void k_dweight(const float* __restrict__ dZ, const float* __restrict__ X, int batch, int I, int O,
                          float* __restrict__ dW, float* __restrict__ db) {
  extern __shared__ float red[];   // [blockDim.x] + [slices]
  const int o = blockIdx.x;
  const int slices = blockDim.x / I;
  const int t = threadIdx.x;
  const int i = t % I, sl = t / I;
  float acc = 0.f, accb = 0.f;
  if (sl < slices) {
    for (int b = sl; b < batch; b += slices) {
      const float g = dZ[(long long)b * O + o];
      acc = fmaf(g, X[(long long)b * I + i], acc);
      if (i == 0) accb += g;
    }
  }
  red[t] = acc;
  float* redb = red + blockDim.x;
  if (i == 0 && sl < slices) redb[sl] = accb;
  __syncthreads();
  if (t < I) {
    float s = 0.f;
    for (int k = 0; k < slices; ++k) s += red[k * I + t];
    dW[(long long)o * I + t] = s;
  }
  if (t == 0) {
    float s = 0.f;
    for (int k = 0; k < slices; ++k) s += redb[k];
    db[o] = s;
  }
}

// dX[b][i] = sum_o dZ[b][o] W[o][i], then times GELU'(Zprev[b][i]) when Zprev != NULL.
__global__ void k_dinput(const float* __restrict__ dZ, const float* __restrict__ W, int batch, int I, int O,
                         const float* __restrict__ Zprev, float* __restrict__ dX) {
  const long long k = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= (long long)batch * I) return;
  const int b = (int)(k / I), i = (int)(k % I);
  const float* g = dZ + (long long)b * O;
  float acc = 0.f;
  for (int o = 0; o < O; ++o) acc = fmaf(g[o], __ldg(W + (long long)o * I + i), acc);
  if (Zprev) acc *= gelu_grad(Zprev[k]);
  dX[k] = acc;
}

__global__ void k_adam(float* __restrict__ p, const float* __restrict__ g, float* __restrict__ m,
                       float* __restrict__ v, long long n, float lr, float b1, float b2, float eps, float wd,
                       float c1, float c2) {
  const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const float gi = g[i];
  const float mi = b1 * m[i] + (1.f - b1) * gi;
  const float vi = b2 * v[i] + (1.f - b2) * gi * gi;
  m[i] = mi;
  v[i] = vi;
  const float mhat = mi / c1, vhat = vi / c2;
  p[i] -= lr * (mhat / (sqrtf(vhat) + eps) + wd * p[i]);
}

// ---- fused forward and backward -----------------------------------------------
struct FusedParams {
  FusedShape s;
  int batch, tiles;
  const float* params;
  const float* X;
  const float* T;
  const float* mask;
  float* Y;            // forward: the outputs
  float* part;         // backward: the CTAs' gradients
  double* sums;        // backward: {loss sum, mask sum} per CTA
};

// All layers of the network on tiles of kFusedRows samples, and the backward
// pass when BWD: the whole step is two launches of a few microseconds, where
// one launch per layer and direction took 17 launches and left most SMs idle
// (a 256-sample step of the 18-64-64-64-56 network: 527 us, of which each
// k_dense read W with a stride of one row per lane). What bounds it now is the
// chain of the layers (each a dot product of up to 128 terms and two CTA
// barriers), so tiles are small: 8 samples give 32 CTAs at a batch of 256.
// A sample's forward sums run in the order of the layer-by-layer path. The
// masked-MSE gradient leaves out the factor 2 / sum(mask), which no CTA knows;
// it is linear, so k_mlp_reduce applies it to the sums.
template <bool BWD>
__global__ void __launch_bounds__(kFusedThreads) k_mlp_fused(const __grid_constant__ FusedParams p) {
  extern __shared__ __align__(16) float sm[];
  constexpr int R = kFusedRows;
  static_assert(R == 8 && kFusedThreads == 256, "the thread maps below");
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  grid_dep_launch_dependents();
  grid_dep_wait();
  const FusedShape S = p.s;
  const int batch = p.batch, out = S.out, ld_dz = S.ld_dz(), tgt = S.tgt();
  // parameters: W rows padded to ld with zeros, biases, mu, sigma (at the start)
  for (int i = tid; i < 2 * S.in; i += kFusedThreads) cp_async4(smem_u32(sm + i), p.params + i);
  for (int l = 0; l <= S.layers; ++l) {
    // 16-byte copies where every row of W starts on 16 bytes, else 4-byte ones,
    // all in flight at once; a thread keeps its column and steps over rows
    const FusedLayer L = S.layer(l);
    const float* W = p.params + L.gw;
    const bool wide = (L.I & 3) == 0 && (reinterpret_cast<uintptr_t>(W) & 15u) == 0;
    if (wide) {
      for (int i = 4 * (tid & 15); i < L.I; i += 64)
#pragma unroll 4
        for (int o = tid >> 4; o < L.O; o += 16) cp_async16(smem_u32(sm + L.w + o * L.ld + i), W + o * L.I + i);
    } else {
      for (int i = lane; i < L.I; i += 32)
#pragma unroll 4
        for (int o = warp; o < L.O; o += 8) cp_async4(smem_u32(sm + L.w + o * L.ld + i), W + o * L.I + i);
    }
    for (int o = tid; o < L.O; o += kFusedThreads) cp_async4(smem_u32(sm + L.b + o), W + L.O * L.I + o);
  }
  // the columns past I of W and of the layer's input are zero
  for (int l = 0; l <= S.layers; ++l) {
    const FusedLayer L = S.layer(l);
    for (int i = L.I + (tid & 7); i < L.ld; i += 8) {
      for (int o = tid >> 3; o < L.O; o += 32) sm[L.w + o * L.ld + i] = 0.f;
      if (tid < 8 * R) sm[L.act + (tid >> 3) * L.ld + i] = 0.f;
    }
  }
  double lsum = 0.0, lcnt = 0.0;
  bool first = true;
  for (int tile = blockIdx.x; tile < p.tiles; tile += gridDim.x, first = false) {
    const int b0 = tile * R;
    const int ny = min(R, batch - b0) * out;   // the tile's rows are contiguous
    // the tile's targets, mask and samples, in flight together (with the
    // parameters, on a CTA's first tile); a thread normalises what it copied
    if constexpr (BWD) {
      for (int k = tid; k < ny; k += kFusedThreads) {
        cp_async4(smem_u32(sm + tgt + k), p.T + (long long)b0 * out + k);
        cp_async4(smem_u32(sm + tgt + R * out + k), p.mask + (long long)b0 * out + k);
      }
    }
    const bool live = b0 + warp < batch;   // a warp a sample
    const FusedLayer L0 = S.layer(0);
    float* xrow = sm + L0.act + warp * L0.ld;
    if (live)
      for (int i = lane; i < S.in; i += 32) cp_async4(smem_u32(xrow + i), p.X + (long long)(b0 + warp) * S.in + i);
    cp_async_wait_all();
    __syncthreads();
    for (int i = lane; i < S.in; i += 32)
      xrow[i] = live ? (xrow[i] - sm[i]) / sm[S.in + i] : 0.f;
    for (int l = 0; l <= S.layers; ++l) {
      const FusedLayer L = S.layer(l);
      const int next_act = S.layer(l + 1).act, next_gp = S.gp(l + 1);   // (not used by the last layer)
      __syncthreads();
      // thread (o, r): output o of samples r and r + 1
      const int r = 2 * (tid >> 6);
      for (int o = tid & 63; o < L.O; o += 64) {
        const float* w = sm + L.w + o * L.ld;
        const float* x = sm + L.act + r * L.ld;
        float z[2] = {sm[L.b + o], sm[L.b + o]};
        // (past I both factors are zeros)
#pragma unroll 4
        for (int i = 0; i < L.I; i += 4) {
          const float4 wv = *reinterpret_cast<const float4*>(w + i);
#pragma unroll
          for (int t = 0; t < 2; ++t) {
            const float4 a = *reinterpret_cast<const float4*>(x + t * L.ld + i);
            z[t] = fmaf(a.x, wv.x, z[t]);
            z[t] = fmaf(a.y, wv.y, z[t]);
            z[t] = fmaf(a.z, wv.z, z[t]);
            z[t] = fmaf(a.w, wv.w, z[t]);
          }
        }
#pragma unroll
        for (int t = 0; t < 2; ++t) {
          const int row = b0 + r + t;
          if (l < S.layers) {
            sm[next_act + (r + t) * S.ldh + o] = gelu(z[t]);
            if constexpr (BWD) sm[next_gp + (r + t) * L.O + o] = gelu_grad(z[t]);
          } else if constexpr (!BWD) {
            if (row < batch) p.Y[(long long)row * out + o] = z[t];
          } else {
            float g = 0.f;
            if (row < batch) {
              const float m = sm[tgt + (R + r + t) * out + o];
              if (m != 0.f) {
                const float tv = sm[tgt + (r + t) * out + o];
                const double d = (double)z[t] - (double)tv;
                lsum += m * d * d;
                lcnt += m;
                g = m * (z[t] - tv);
              }
            }
            sm[S.dz() + (r + t) * ld_dz + o] = g;
          }
        }
      }
    }
    if constexpr (BWD) {
      int cur = S.dz(), nxt = cur + R * ld_dz;
      for (int l = S.layers; l >= 0; --l) {
        const FusedLayer L = S.layer(l);
        const int O4 = (L.O + 3) >> 2, I4 = (L.I + 3) >> 2;
        __syncthreads();
        // the quad past O of dZ (read below, its sums land in padding)
        float* part = p.part + (long long)blockIdx.x * S.part_floats() + L.gpart;
        // dW: an item is 4 outputs x 4 inputs, summed over the tile's samples
        for (int oq = tid >> 4; oq < O4; oq += 16) for (int iq = tid & 15; iq < I4; iq += 16) {
          float acc[4][4];
#pragma unroll
          for (int a = 0; a < 4; ++a)
#pragma unroll
            for (int b = 0; b < 4; ++b) acc[a][b] = 0.f;
#pragma unroll
          for (int r = 0; r < R; ++r) {
            const float4 g = *reinterpret_cast<const float4*>(sm + cur + r * ld_dz + 4 * oq);
            const float4 x = *reinterpret_cast<const float4*>(sm + L.act + r * L.ld + 4 * iq);
            const float gs[4] = {g.x, g.y, g.z, g.w}, xs[4] = {x.x, x.y, x.z, x.w};
#pragma unroll
            for (int a = 0; a < 4; ++a)
#pragma unroll
              for (int b = 0; b < 4; ++b) acc[a][b] = fmaf(gs[a], xs[b], acc[a][b]);
          }
#pragma unroll
          for (int a = 0; a < 4; ++a) {
            float4* q = reinterpret_cast<float4*>(part + (long long)(4 * oq + a) * (4 * I4) + 4 * iq);
            float4 v = make_float4(acc[a][0], acc[a][1], acc[a][2], acc[a][3]);
            if (!first) {
              const float4 w = *q;
              v = make_float4(v.x + w.x, v.y + w.y, v.z + w.z, v.w + w.w);
            }
            *q = v;
          }
        }
        float* bpart = part + (long long)(4 * O4) * (4 * I4);
        for (int o = tid; o < L.O; o += kFusedThreads) {
          float s = 0.f;
#pragma unroll
          for (int r = 0; r < R; ++r) s += sm[cur + r * ld_dz + o];
          bpart[o] = first ? s : bpart[o] + s;
        }
        if (l > 0) {
          // dX = (dZ W) * GELU': input i of samples r and r + 1
          const int r = 2 * (tid >> 6);
          const float* gp = sm + S.gp(l) + r * L.I;
          for (int i = tid & 63; i < L.I; i += 64) {
            const float* g = sm + cur + r * ld_dz;
            const float* w = sm + L.w + i;
            float a[2] = {0.f, 0.f};
            int o = 0;
#pragma unroll 4
            for (; o + 4 <= L.O; o += 4) {
              const float w0 = w[o * L.ld], w1 = w[(o + 1) * L.ld], w2 = w[(o + 2) * L.ld], w3 = w[(o + 3) * L.ld];
#pragma unroll
              for (int t = 0; t < 2; ++t) {
                const float4 gv = *reinterpret_cast<const float4*>(g + t * ld_dz + o);
                a[t] = fmaf(gv.x, w0, a[t]);
                a[t] = fmaf(gv.y, w1, a[t]);
                a[t] = fmaf(gv.z, w2, a[t]);
                a[t] = fmaf(gv.w, w3, a[t]);
              }
            }
            for (; o < L.O; ++o)
#pragma unroll
              for (int t = 0; t < 2; ++t) a[t] = fmaf(g[t * ld_dz + o], w[o * L.ld], a[t]);
#pragma unroll
            for (int t = 0; t < 2; ++t) sm[nxt + (r + t) * ld_dz + i] = a[t] * gp[t * L.I + i];
          }
          const int t = cur;
          cur = nxt;
          nxt = t;
        }
      }
    }
    __syncthreads();   // the next tile's copies overwrite what this one reads
  }
  if constexpr (BWD) {
    __shared__ double red[2][kFusedThreads / 32];
    for (int o = 16; o; o >>= 1) {
      lsum += __shfl_xor_sync(0xffffffffu, lsum, o);
      lcnt += __shfl_xor_sync(0xffffffffu, lcnt, o);
    }
    if ((tid & 31) == 0) {
      red[0][tid >> 5] = lsum;
      red[1][tid >> 5] = lcnt;
    }
    __syncthreads();
    if (tid < 2) {
      double s = 0.0;
      for (int w = 0; w < kFusedThreads / 32; ++w) s += red[tid][w];
      p.sums[2 * blockIdx.x + tid] = s;
    }
  }
}

struct ReduceParams {
  FusedShape s;
  int ctas;
  const float* part;
  const double* sums;
  float* grad;
  float* loss;
};

// grad = 2 / sum(mask) * (the CTAs' gradients, added in a fixed order): blockIdx.y
// is the layer, a thread one weight or bias of it. mu and sigma are not
// trained: their gradient is zero.
__global__ void __launch_bounds__(128) k_mlp_reduce(const __grid_constant__ ReduceParams p) {
  __shared__ double tot[2];
  grid_dep_launch_dependents();
  grid_dep_wait();
  const int l = blockIdx.y;
  const FusedLayer L = p.s.layer(l);
  const int I = L.I, O = L.O, I4 = (I + 3) & ~3, O4 = (O + 3) & ~3, stride = p.s.part_floats();
  const int k = blockIdx.x * blockDim.x + threadIdx.x;
  const bool is_w = k < O * I, is_b = !is_w && k < O * I + O;
  float s = 0.f;
  if (is_w || is_b) {
    const float* q = p.part + L.gpart + (is_w ? (k / I) * I4 + k % I : O4 * I4 + (k - O * I));
    for (int c0 = 0; c0 < p.ctas; c0 += 16) {
      // 16 CTAs' sums in pairs: 12 roundings deep for 128 CTAs, not 128
      float v[16];
#pragma unroll
      for (int c = 0; c < 16; ++c) v[c] = c0 + c < p.ctas ? q[(long long)(c0 + c) * stride] : 0.f;
#pragma unroll
      for (int d = 1; d < 16; d *= 2)
#pragma unroll
        for (int c = 0; c < 16; c += 2 * d) v[c] += v[c + d];
      s += v[0];
    }
  }
  if (threadIdx.x < 64) {
    // lanes add every 32nd CTA's sum, then a fixed tree: one order for all
    const int which = threadIdx.x >> 5, lane = threadIdx.x & 31;
    double v = 0.0;
    for (int c = lane; c < p.ctas; c += 32) v += p.sums[2 * c + which];
    for (int o = 16; o; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    if (lane == 0) tot[which] = v;
  }
  __syncthreads();
  const double total = tot[1] > 0 ? tot[1] : 1.0;
  if (is_w || is_b) p.grad[L.gw + k] = (float)(2.0 / total * s);   // the factor rounds once, with the product
  if (l == 0 && k < 2 * p.s.in) p.grad[k] = 0.f;
  if (l == 0 && k == 0 && p.loss) *p.loss = (float)(tot[0] / total);
}

bool aligned_to(const void* q, uintptr_t a) { return (reinterpret_cast<uintptr_t>(q) % a) == 0; }

// The fused step's launches. Forward: Y; backward: grad and loss, with `work`
// (16-byte aligned, fused_ws floats) for the CTAs' sums.
spmm_status launch_fused(const Layout& L, const float* params, const float* X, const float* T, const float* mask,
                         int batch, float* Y, float* grad, float* loss, float* work, cudaStream_t s) {
  const FusedShape S = L.fused_shape();
  FusedParams p;
  std::memset(&p, 0, sizeof(p));
  p.s = S;
  p.params = params;
  p.X = X;
  p.T = T;
  p.mask = mask;
  p.Y = Y;
  p.batch = batch;
  p.tiles = (batch + kFusedRows - 1) / kFusedRows;
  const int smem = S.smem_floats() * (int)sizeof(float);
  const int ctas = L.fused_ctas(batch);
  if (grad) {
    p.sums = reinterpret_cast<double*>(work);
    p.part = work + 4LL * ctas;
  }
  const void* fn = grad ? reinterpret_cast<const void*>(&k_mlp_fused<true>) : reinterpret_cast<const void*>(&k_mlp_fused<false>);
  // one limit for all networks: the attribute is per kernel, not per launch
  SPMM_CUDA_TRY(ensure_smem_attr(fn, (int)kFusedSmemMax));
  if (!grad) {
    SPMM_CUDA_TRY(launch_kernel(&k_mlp_fused<false>, dim3((unsigned)ctas), dim3(kFusedThreads), (size_t)smem, s, p));
    return SPMM_OK;
  }
  SPMM_CUDA_TRY(launch_kernel(&k_mlp_fused<true>, dim3((unsigned)ctas), dim3(kFusedThreads), (size_t)smem, s, p));
  ReduceParams r;
  std::memset(&r, 0, sizeof(r));
  r.s = S;
  r.ctas = ctas;
  r.part = p.part;
  r.sums = p.sums;
  r.grad = grad;
  r.loss = loss;
  int most = 2 * L.in;
  for (int l = 0; l <= L.layers; ++l) most = std::max(most, L.fan_out(l) * (L.fan_in(l) + 1));
  SPMM_CUDA_TRY(launch_kernel(&k_mlp_reduce, dim3((unsigned)((most + 127) / 128), (unsigned)(L.layers + 1)), dim3(128),
                              (size_t)0, s, r));
  return SPMM_OK;
}

inline unsigned blocks_for(long long n, int t) { return (unsigned)((n + t - 1) / t); }

// Forward pass into the workspace; returns the pointer to Y inside it.
spmm_status forward_ws(const Layout& L, const float* params, const float* X, int batch, float* ws,
                       cudaStream_t s, float** Y_out) {
  float* Xn = ws;
  float* cur = Xn;
  k_normalize<<<blocks_for((long long)batch * L.in, 256), 256, 0, s>>>(X, params, params + L.in, batch, L.in, Xn);
  float* p = Xn + (long long)batch * L.in;
  for (int l = 0; l <= L.layers; ++l) {
    const int I = L.fan_in(l), O = L.fan_out(l);
    float* Z = p;
    float* A = l < L.layers ? p + (long long)batch * O : nullptr;
    const size_t sm = (size_t)64 * I * sizeof(float);
    k_dense<<<blocks_for(batch, 64), 256, sm, s>>>(cur, params + L.w_off(l), params + L.b_off(l), batch, I, O, Z,
                                                   A);
    if (l < L.layers) {
      cur = A;
      p += 2LL * batch * O;
    } else {
      *Y_out = Z;
    }
  }
  SPMM_CUDA_TRY(cudaGetLastError());
  return SPMM_OK;
}

}  // namespace
}  // namespace spmm

using namespace spmm;

struct spmm_cost_model {
  spmm_mlp_shape shape;
  float* d_params = nullptr;
  float* d_ws = nullptr;    // workspace for a batch of one
  float* d_x = nullptr;
  int device = -1;
};

extern "C" {

long long spmm_mlp_param_count(const spmm_mlp_shape* shape) {
  return valid(shape) ? layout(shape).params() : -1;
}

long long spmm_mlp_workspace_floats(const spmm_mlp_shape* shape, int batch) {
  return valid(shape) && batch > 0 ? layout(shape).ws(batch) : -1;
}

spmm_status spmm_mlp_forward(const spmm_mlp_shape* shape, const float* params, const float* X, int batch,
                             float* Y, float* work, void* stream) {
  if (!valid(shape) || !params || !X || !Y || !work || batch <= 0)
    return fail(SPMM_ERR_INVALID_ARG, "bad MLP forward arguments");
  const Layout L = layout(shape);
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  if (L.fused()) return launch_fused(L, params, X, nullptr, nullptr, batch, Y, nullptr, nullptr, work, s);
  float* Yw = nullptr;
  spmm_status st = forward_ws(L, params, X, batch, work, s, &Yw);
  if (st != SPMM_OK) return st;
  SPMM_CUDA_TRY(cudaMemcpyAsync(Y, Yw, sizeof(float) * batch * L.out, cudaMemcpyDeviceToDevice, s));
  return SPMM_OK;
}

spmm_status spmm_mlp_backward(const spmm_mlp_shape* shape, const float* params, const float* X, const float* T,
                              const float* mask, int batch, float* grad, float* loss, float* work, void* stream) {
  if (!valid(shape) || !params || !X || !T || !mask || !grad || !work || batch <= 0)
    return fail(SPMM_ERR_INVALID_ARG, "bad MLP backward arguments");
  const Layout L = layout(shape);
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  if (L.fused() && aligned_to(work, 16)) return launch_fused(L, params, X, T, mask, batch, nullptr, grad, loss, work, s);
  float* Y = nullptr;
  spmm_status st = forward_ws(L, params, X, batch, work, s, &Y);
  if (st != SPMM_OK) return st;
  const int wmax = L.hidden > L.out ? L.hidden : L.out;
  float* g0 = Y + (long long)batch * L.out;
  float* g1 = g0 + (long long)batch * wmax;
  SPMM_CUDA_TRY(cudaMemsetAsync(grad, 0, sizeof(float) * L.norm_floats(), s));
  k_mse<<<1, 1024, 0, s>>>(Y, T, mask, (long long)batch * L.out, g0, loss);
  // layer l's input activation: Xn for l = 0, else A_{l-1}; its pre-activation Z_{l-1}
  auto act_in = [&](int l) -> const float* {
    if (l == 0) return work;
    return work + (long long)batch * L.in + (2LL * (l - 1) + 1) * batch * L.hidden;
  };
  auto z_of = [&](int l) -> const float* {   // Z of hidden layer l
    return work + (long long)batch * L.in + 2LL * l * batch * L.hidden;
  };
  float* dZ = g0;
  float* dX = g1;
  for (int l = L.layers; l >= 0; --l) {
    const int I = L.fan_in(l), O = L.fan_out(l);
    const int slices = 256 / I > 0 ? 256 / I : 1;
    const int threads = slices * I <= 1024 ? slices * I : I;
    k_dweight<<<O, threads, sizeof(float) * (threads + slices), s>>>(dZ, act_in(l), batch, I, O,
                                                                     grad + L.w_off(l), grad + L.b_off(l));
    if (l > 0) {
      k_dinput<<<blocks_for((long long)batch * I, 256), 256, 0, s>>>(dZ, params + L.w_off(l), batch, I, O,
                                                                     z_of(l - 1), dX);
      float* t = dZ;
      dZ = dX;
      dX = t;
    }
  }
  SPMM_CUDA_TRY(cudaGetLastError());
  return SPMM_OK;
}

spmm_status spmm_mlp_adam(float* params, const float* grad, float* m, float* v, long long n, long long offset,
                          float lr, float beta1, float beta2, float eps, float weight_decay, int step,
                          void* stream) {
  if (!params || !grad || !m || !v || n <= 0 || offset < 0 || offset >= n || step < 1)
    return fail(SPMM_ERR_INVALID_ARG, "bad Adam arguments");
  const long long cnt = n - offset;
  const float c1 = 1.f - powf(beta1, (float)step), c2 = 1.f - powf(beta2, (float)step);
  k_adam<<<blocks_for(cnt, 256), 256, 0, static_cast<cudaStream_t>(stream)>>>(
      params + offset, grad + offset, m + offset, v + offset, cnt, lr, beta1, beta2, eps, weight_decay, c1, c2);
  SPMM_CUDA_TRY(cudaGetLastError());
  return SPMM_OK;
}

spmm_status spmm_cost_model_create(const spmm_mlp_shape* shape, const float* host_params,
                                   spmm_cost_model** out) {
  if (!out) return fail(SPMM_ERR_INVALID_ARG, "null output");
  *out = nullptr;
  if (!valid(shape) || !host_params) return fail(SPMM_ERR_INVALID_ARG, "bad cost model arguments");
  if (shape->out != spmm_tune_config_count())
    return fail(SPMM_ERR_INVALID_ARG, "the model must predict one time per tuner configuration");
  const Layout L = layout(shape);
  spmm_cost_model* m = new spmm_cost_model();
  m->shape = *shape;
  cudaGetDevice(&m->device);
  cudaError_t ce = cudaMalloc(&m->d_params, sizeof(float) * L.params());
  if (ce == cudaSuccess)
    ce = cudaMemcpy(m->d_params, host_params, sizeof(float) * L.params(), cudaMemcpyHostToDevice);
  if (ce == cudaSuccess) ce = cudaMalloc(&m->d_ws, sizeof(float) * L.ws(1));
  if (ce == cudaSuccess) ce = cudaMalloc(&m->d_x, sizeof(float) * (L.in + L.out));
  if (ce != cudaSuccess) {
    spmm_cost_model_destroy(m);
    return cuda_fail(ce, "creating the cost model");
  }
  *out = m;
  return SPMM_OK;
}

spmm_status spmm_cost_model_load(const char* path, spmm_cost_model** out) {
  if (!path || !out) return fail(SPMM_ERR_INVALID_ARG, "null argument");
  *out = nullptr;
  FILE* f = std::fopen(path, "rb");
  if (!f) return fail(SPMM_ERR_INVALID_ARG, std::string("cannot open ") + path);
  char magic[8];
  int32_t dims[4];
  bool ok = std::fread(magic, 1, 8, f) == 8 && std::memcmp(magic, "SPMMCM01", 8) == 0 &&
            std::fread(dims, sizeof(int32_t), 4, f) == 4;
  spmm_mlp_shape s{dims[0], dims[1], dims[2], dims[3]};
  std::vector<float> params;
  if (ok && valid(&s)) {
    params.resize((size_t)layout(&s).params());
    ok = std::fread(params.data(), sizeof(float), params.size(), f) == params.size();
  } else {
    ok = false;
  }
  std::fclose(f);
  if (!ok) return fail(SPMM_ERR_INVALID_ARG, std::string("not a cost model file: ") + path);
  return spmm_cost_model_create(&s, params.data(), out);
}

spmm_status spmm_cost_model_destroy(spmm_cost_model* m) {
  if (!m) return SPMM_OK;
  if (m->d_params) cudaFree(m->d_params);
  if (m->d_ws) cudaFree(m->d_ws);
  if (m->d_x) cudaFree(m->d_x);
  delete m;
  return SPMM_OK;
}

spmm_status spmm_cost_model_select(const spmm_cost_model* m, const spmm_bcsr_desc* A, int N, spmm_config* out,
                                   float* predicted, void* stream) {
  if (!m || !A || !out) return fail(SPMM_ERR_INVALID_ARG, "null argument");
  const Layout L = layout(&m->shape);
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  if (L.in != SPMM_FEATURES) return fail(SPMM_ERR_INVALID_ARG, "the model's input must be the structure features");
  std::vector<float> f(SPMM_FEATURES, 0.f), y(L.out);
  spmm_status st = spmm_structure_features(A, N, f.data(), stream);
  if (st != SPMM_OK) return st;
  SPMM_CUDA_TRY(cudaMemcpyAsync(m->d_x, f.data(), sizeof(float) * L.in, cudaMemcpyHostToDevice, s));
  float* Y = m->d_x + L.in;
  if (L.fused())
    st = launch_fused(L, m->d_params, m->d_x, nullptr, nullptr, 1, Y, nullptr, nullptr, nullptr, s);
  else
    st = forward_ws(L, m->d_params, m->d_x, 1, m->d_ws, s, &Y);
  if (st != SPMM_OK) return st;
  SPMM_CUDA_TRY(cudaMemcpyAsync(y.data(), Y, sizeof(float) * L.out, cudaMemcpyDeviceToHost, s));
  SPMM_CUDA_TRY(cudaStreamSynchronize(s));
  int best = -1;
  for (int i = 0; i < L.out; ++i) {
    spmm_config c;
    spmm_tune_config(i, &c);
    const bool ok = spmm_config_supported(A->bR, A->dtype, N, &c) == SPMM_OK;
    if (predicted) predicted[i] = ok ? std::exp(y[i]) * 1e-3f : INFINITY;   // outputs are ln(microseconds)
    if (ok && (best < 0 || y[i] < y[best])) best = i;
  }
  if (best < 0) return fail(SPMM_ERR_UNSUPPORTED, "no configuration runs this product");
  return spmm_tune_config(best, out);
}

}  // extern "C"
