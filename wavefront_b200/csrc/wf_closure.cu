// wf_closure.cu -- the learned thin-CPML boundary closure (no reference
// counterpart): a per-face 3-layer 3D convolutional network that corrects
// the fields in the 8-cell band next to each face of a grid with a thin
// (4-cell) CPML, so that it behaves like a thick one.
//
// Tensors are "band" tensors [N][C][D=8][H][W]: sample n (a face, or a crop
// of one), channel c, distance d from the outer face (0 = outermost cell),
// and the two tangential coordinates in increasing axis order.  Every conv
// is 3x3x3, stride 1, zero padding, no bias; weights are bfloat16
// [F][Co][Ci][27] (F = 6 faces; sample n uses face[n]) and every sum
// accumulates in FP32.  GELU is the erf form 0.5 z (1 + erf(z / sqrt 2)).
//
// Training runs on these kernels too: forward (keeping pre-activations),
// backward to the input and to the weights, GELU backward, the MSE loss and
// its gradient, and Adam on FP32 master weights with a bfloat16 copy for
// the forward pass.
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include <algorithm>

#include "wf_band.cuh"
#include "wf_closure.h"

namespace wf {

namespace {

constexpr int kMaxC = 16;       // channels per layer at most
constexpr int kTaps = 27;
constexpr float kInvSqrt2 = 0.70710678118654752f;
constexpr float kInvSqrt2Pi = 0.39894228040143268f;

__device__ __forceinline__ float gelu(float z) { return 0.5f * z * (1.0f + erff(z * kInvSqrt2)); }
__device__ __forceinline__ float gelu_grad(float z) {
  return 0.5f * (1.0f + erff(z * kInvSqrt2)) + z * kInvSqrt2Pi * expf(-0.5f * z * z);
}

// out[n][co][p] = sum_ci sum_tap w[face[n]][co][ci][tap] * in[n][ci][p + tap]
// (one thread per output voxel, all output channels in registers; the
// sample's weights staged in shared memory as FP32)
__global__ void k_conv_fwd(const float *in, const __nv_bfloat16 *w, const int *face, float *z,
                           float *a, int n, int ci, int co, int D, int H, int W, int act) {
  extern __shared__ float s_w[];  // [co][ci][27] of the block's sample
  const long long P = static_cast<long long>(D) * H * W;
  const int s = blockIdx.y;       // sample
  const int f = face ? face[s] : 0;
  const int nw = co * ci * kTaps;
  for (int i = threadIdx.x; i < nw; i += blockDim.x)
    s_w[i] = __bfloat162float(w[static_cast<long long>(f) * nw + i]);
  __syncthreads();
  const long long p = static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x;
  if (p >= P || s >= n) return;
  const int x = static_cast<int>(p % W), y = static_cast<int>((p / W) % H), d = static_cast<int>(p / (static_cast<long long>(W) * H));
  float acc[kMaxC];
#pragma unroll
  for (int o = 0; o < kMaxC; ++o) acc[o] = 0.0f;
  const float *src = in + static_cast<long long>(s) * ci * P;
  for (int c = 0; c < ci; ++c) {
    const float *sc = src + c * P;
    for (int t = 0; t < kTaps; ++t) {
      const int dd = d + t / 9 - 1, yy = y + (t / 3) % 3 - 1, xx = x + t % 3 - 1;
      if (dd < 0 || dd >= D || yy < 0 || yy >= H || xx < 0 || xx >= W) continue;
      const float v = sc[(static_cast<long long>(dd) * H + yy) * W + xx];
#pragma unroll
      for (int o = 0; o < kMaxC; ++o)
        if (o < co) acc[o] = __fmaf_rn(s_w[(o * ci + c) * kTaps + t], v, acc[o]);
    }
  }
  for (int o = 0; o < co; ++o) {
    const long long k = (static_cast<long long>(s) * co + o) * P + p;
    if (z) z[k] = acc[o];
    a[k] = act ? gelu(acc[o]) : acc[o];
  }
}

// The same convolution for the network's output-channel counts (CO = 16, 6),
// blocked for the FMA pipes: a thread computes 4 consecutive voxels of one
// row from 6 staged inputs per (channel, dz, dy), and the weights sit in
// shared memory output-channel fastest ([ci][27][CP], CP = CO rounded up to
// 4, zero padded) so that 128-bit loads feed CO FMAs for each of the 4
// voxels.  Every voxel still sums channel by channel and tap by tap in the
// order of k_conv_fwd, skipping the same out-of-range taps, so the results
// are identical.
template <int CO>
__global__ void __launch_bounds__(128) k_conv_fwd4(const float *in, const __nv_bfloat16 *w,
                                                   const int *face, float *z, float *a, int n,
                                                   int ci, int D, int H, int W, int act) {
  constexpr int CP = (CO + 3) / 4 * 4;
  extern __shared__ float s_w[];  // [ci][27][CP] of the block's sample
  const int s = blockIdx.y;
  const int f = face ? face[s] : 0;
  const int nw = ci * kTaps * CP;
  for (int i = threadIdx.x; i < nw; i += blockDim.x) {
    const int o = i % CP, ct = i / CP;  // ct = c * 27 + t
    const int c = ct / kTaps, t = ct % kTaps;
    s_w[i] = o < CO ? __bfloat162float(w[((static_cast<long long>(f) * CO + o) * ci + c) * kTaps + t])
                    : 0.0f;
  }
  __syncthreads();
  const int QW = (W + 3) / 4;
  const long long q = static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x;
  if (q >= static_cast<long long>(D) * H * QW || s >= n) return;
  const int x0 = static_cast<int>(q % QW) * 4, y = static_cast<int>((q / QW) % H),
            d = static_cast<int>(q / (static_cast<long long>(QW) * H));
  bool ok[6];  // input column x0 - 1 + k inside the row
#pragma unroll
  for (int k = 0; k < 6; ++k) ok[k] = x0 - 1 + k >= 0 && x0 - 1 + k < W;
  float acc[4][CO];
#pragma unroll
  for (int v = 0; v < 4; ++v)
#pragma unroll
    for (int o = 0; o < CO; ++o) acc[v][o] = 0.0f;
  const long long P = static_cast<long long>(D) * H * W;
  const float *src = in + static_cast<long long>(s) * ci * P;
  for (int c = 0; c < ci; ++c) {
    const float *sc = src + c * P;
    for (int dz = -1; dz <= 1; ++dz) {
      const int dd = d + dz;
      if (dd < 0 || dd >= D) continue;
      for (int dy = -1; dy <= 1; ++dy) {
        const int yy = y + dy;
        if (yy < 0 || yy >= H) continue;
        const float *row = sc + (static_cast<long long>(dd) * H + yy) * W + x0 - 1;
        float r[6];
#pragma unroll
        for (int k = 0; k < 6; ++k) r[k] = ok[k] ? __ldg(row + k) : 0.0f;
        const float *wt = s_w + (c * kTaps + (dz + 1) * 9 + (dy + 1) * 3) * CP;
#pragma unroll
        for (int dx = 0; dx < 3; ++dx) {
          float wv[CP];
#pragma unroll
          for (int o4 = 0; o4 < CP / 4; ++o4) {
            const float4 w4 = *reinterpret_cast<const float4 *>(wt + dx * CP + 4 * o4);
            wv[4 * o4] = w4.x;
            wv[4 * o4 + 1] = w4.y;
            wv[4 * o4 + 2] = w4.z;
            wv[4 * o4 + 3] = w4.w;
          }
#pragma unroll
          for (int v = 0; v < 4; ++v) {
            if (!ok[v + dx]) continue;  // the tap k_conv_fwd skips
#pragma unroll
            for (int o = 0; o < CO; ++o) acc[v][o] = __fmaf_rn(wv[o], r[v + dx], acc[v][o]);
          }
        }
      }
    }
  }
#pragma unroll
  for (int v = 0; v < 4; ++v) {
    if (x0 + v >= W) break;
    const long long p = (static_cast<long long>(d) * H + y) * W + x0 + v;
#pragma unroll
    for (int o = 0; o < CO; ++o) {
      const long long k = (static_cast<long long>(s) * CO + o) * P + p;
      if (z) z[k] = acc[v][o];
      a[k] = act ? gelu(acc[v][o]) : acc[v][o];
    }
  }
}

// din[n][ci][p] = sum_co sum_tap w[co][ci][tap] * dz[n][co][p - tap]
__global__ void k_conv_bwd_data(const float *dz, const __nv_bfloat16 *w, const int *face, float *din,
                                int n, int ci, int co, int D, int H, int W) {
  extern __shared__ float s_w[];
  const long long P = static_cast<long long>(D) * H * W;
  const int s = blockIdx.y;
  const int f = face ? face[s] : 0;
  const int nw = co * ci * kTaps;
  for (int i = threadIdx.x; i < nw; i += blockDim.x)
    s_w[i] = __bfloat162float(w[static_cast<long long>(f) * nw + i]);
  __syncthreads();
  const long long p = static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x;
  if (p >= P || s >= n) return;
  const int x = static_cast<int>(p % W), y = static_cast<int>((p / W) % H), d = static_cast<int>(p / (static_cast<long long>(W) * H));
  float acc[kMaxC];
#pragma unroll
  for (int c = 0; c < kMaxC; ++c) acc[c] = 0.0f;
  const float *src = dz + static_cast<long long>(s) * co * P;
  for (int o = 0; o < co; ++o) {
    const float *so = src + o * P;
    for (int t = 0; t < kTaps; ++t) {
      const int dd = d - (t / 9 - 1), yy = y - ((t / 3) % 3 - 1), xx = x - (t % 3 - 1);
      if (dd < 0 || dd >= D || yy < 0 || yy >= H || xx < 0 || xx >= W) continue;
      const float g = so[(static_cast<long long>(dd) * H + yy) * W + xx];
#pragma unroll
      for (int c = 0; c < kMaxC; ++c)
        if (c < ci) acc[c] = __fmaf_rn(s_w[(o * ci + c) * kTaps + t], g, acc[c]);
    }
  }
  for (int c = 0; c < ci; ++c) din[(static_cast<long long>(s) * ci + c) * P + p] = acc[c];
}

// The sum of tap t's products over the voxels [d0,d1) x [y0,y1) x [x0,x1) of
// one sample's channels, the taps outside the planes left out.  The staged
// kernels multiply their zero halo instead, which only an infinity or a NaN on
// the other side turns into something else: a sum that is not finite is taken
// again here.
__device__ float bw_checked(const float *v, const float *g, int t, int d0, int d1, int y0, int y1,
                            int x0, int x1, int D, int H, int W, float sum) {
  const int od = t / 9 - 1, oy = t / 3 % 3 - 1, ox = t % 3 - 1;
  for (int d = max(d0, -od); d < min(d1, D - od); ++d)
    for (int y = max(y0, -oy); y < min(y1, H - oy); ++y) {
      const float *gr = g + (static_cast<long long>(d) * H + y) * W;
      const float *vr = v + (static_cast<long long>(d + od) * H + y + oy) * W + ox;
      for (int x = max(x0, -ox); x < min(x1, W - ox); ++x) sum = __fmaf_rn(gr[x], vr[x], sum);
    }
  return sum;
}
__device__ __forceinline__ bool not_finite(float v) { return !(fabsf(v) <= 3.402823466e38f); }

// dw[face][co][ci][tap] += sum over samples of that face and voxels p of
// dz[n][co][p] * in[n][ci][p + tap], for samples of few voxels: one thread per
// weight, the samples split over blockIdx.y, both operands from global memory.
// The tiles below cost 16 to 18 us however little there is to sum (their
// unrolled code is fetched once and run once): 1 sample of 8 x 8, 16 -> 16
// channels, takes 11.6 us here and 17.8 there, 63 of 4 x 4 15 and 32; at 128
// voxels a sample the two are equal.
constexpr int kBwFewVoxels = 128;
__global__ void k_conv_bwd_weight_few(const float *in, const float *dz, const int *face, float *dw, int n,
                                      int ci, int co, int D, int H, int W, int nface) {
  const int nw = co * ci * kTaps, e = blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= nw) return;
  const int o = e / (ci * kTaps), c = (e / kTaps) % ci, t = e % kTaps;
  const long long P = static_cast<long long>(D) * H * W;
  float acc[8];  // by face
  for (float &a : acc) a = 0.0f;
  for (int s = blockIdx.y; s < n; s += gridDim.y) {
    const int f = face ? face[s] : 0;
    if (f < 0 || f >= nface) continue;
    acc[f] += bw_checked(in + (static_cast<long long>(s) * ci + c) * P, dz + (static_cast<long long>(s) * co + o) * P,
                         t, 0, D, 0, H, 0, W, D, H, W, 0.0f);
  }
  for (int f = 0; f < nface; ++f)
    if (acc[f] != 0.0f) atomicAdd(dw + static_cast<long long>(f) * nw + e, acc[f]);
}

// The same from tiles in shared memory.
//
// A CTA works for one face (blockIdx.y) on every gridDim.x-th tile of the
// face's samples: 4 planes x 4 rows x 16 columns of dz and their haloed input
// in shared memory.  A thread owns one input channel, two output channels and
// all 27 taps (54 sums kept in registers over all its tiles): a row of 4
// columns takes one 128-bit load per output channel and two per tap row for
// 216 FMAs, so the FMA pipes bound it.  Threads beyond ci * co / 2 split the
// tile's rows between them; the sums meet in global memory once per CTA.
// Measured on B200 (a training step on 128 samples of 8 x 16 x 16): 4.37 ms, of
// which the three layers' weight gradients took 0.69 + 1.59 + 1.44 ms with one
// thread per weight reading both operands from global memory; 145 us a layer now.
constexpr int kBwD = 4, kBwY = 4, kBwX = 16;         // tile of dz
constexpr int kBwRow = 20;                           // input row: 18 columns, 16-byte pitch
constexpr int kBwIn = (kBwD + 2) * (kBwY + 2) * kBwRow + 4;  // one input channel; + 4: channels
constexpr int kBwDz = kBwD * kBwY * kBwX + 4;                // start in different banks
constexpr int kBwSmem = 16 * (kBwIn + kBwDz) * 4;
constexpr int kBwThreads = 256;

__global__ void __launch_bounds__(kBwThreads, 2)
    k_conv_bwd_weight(const float *in, const float *dz, const int *face, float *dw, int n, int ci,
                      int co, int D, int H, int W) {
  extern __shared__ __align__(16) float s_t[];
  float *s_in = s_t, *s_dz = s_t + 16 * kBwIn;
  const int f = blockIdx.y, tid = threadIdx.x, lane = tid & 31;
  const int co2 = (co + 1) / 2, combos = ci * co2, parts = kBwThreads / combos;
  const int combo = tid % combos, part = tid / combos;
  const int c = combo % ci, o = 2 * (combo / ci);
  const bool active = part < parts;
  const int tx = (W + kBwX - 1) / kBwX, ty = (H + kBwY - 1) / kBwY, td = (D + kBwD - 1) / kBwD;
  const int tiles = tx * ty * td;
  const long long P = static_cast<long long>(D) * H * W;
  float acc0[27], acc1[27];
#pragma unroll
  for (int t = 0; t < 27; ++t) acc0[t] = acc1[t] = 0.0f;
  bool any = false;
  long long count = 0;  // tiles of this face so far
  for (int s0 = 0; s0 < n; s0 += 32) {
    const int mine = s0 + lane < n ? (face ? face[s0 + lane] : 0) : -1;
    for (unsigned m = __ballot_sync(0xffffffffu, mine == f); m; m &= m - 1, count += tiles) {
      const int s = s0 + __ffs(m) - 1;
      // this CTA's tiles of the sample: those with (count + q) % gridDim.x == blockIdx.x
      int q = static_cast<int>((blockIdx.x + gridDim.x - count % gridDim.x) % gridDim.x);
      for (; q < tiles; q += gridDim.x) {
        const int x0 = q % tx * kBwX, y0 = q / tx % ty * kBwY, d0 = q / (tx * ty) * kBwD;
        any = true;
        __syncthreads();  // the tile before is consumed
        const float *src = in + static_cast<long long>(s) * ci * P;
        // 16 lanes a row; the two halo columns after
        constexpr int kRows = (kBwD + 2) * (kBwY + 2);
        const int k = tid & 15;
#pragma unroll 6
        for (int i = tid >> 4; i < ci * kRows; i += kBwThreads / 16) {
          const int ch = i / kRows, row = i % kRows;
          const int d = d0 - 1 + row / (kBwY + 2), y = y0 - 1 + row % (kBwY + 2), x = x0 + k;
          const bool ok = d >= 0 && d < D && y >= 0 && y < H && x < W;
          s_in[ch * kBwIn + row * kBwRow + 1 + k] =
              ok ? __ldg(src + ch * P + (static_cast<long long>(d) * H + y) * W + x) : 0.0f;
        }
        for (int i = tid; i < 2 * ci * kRows; i += kBwThreads) {
          const int side = i & 1, ch = (i >> 1) / kRows, row = (i >> 1) % kRows;
          const int d = d0 - 1 + row / (kBwY + 2), y = y0 - 1 + row % (kBwY + 2),
                    x = side ? x0 + kBwX : x0 - 1;
          const bool ok = d >= 0 && d < D && y >= 0 && y < H && x >= 0 && x < W;
          s_in[ch * kBwIn + row * kBwRow + side * (kBwX + 1)] =
              ok ? __ldg(src + ch * P + (static_cast<long long>(d) * H + y) * W + x) : 0.0f;
        }
        const float *g = dz + static_cast<long long>(s) * co * P;
#pragma unroll 4
        for (int i = tid >> 4; i < 2 * co2 * kBwD * kBwY; i += kBwThreads / 16) {
          const int ch = i / (kBwD * kBwY), row = i % (kBwD * kBwY);
          const int d = d0 + row / kBwY, y = y0 + row % kBwY, x = x0 + k;
          const bool ok = ch < co && d < D && y < H && x < W;
          s_dz[ch * kBwDz + row * kBwX + k] =
              ok ? __ldg(g + ch * P + (static_cast<long long>(d) * H + y) * W + x) : 0.0f;
        }
        __syncthreads();
        if (!active) continue;
        // rows and columns of padding add zeros: left out
        const int xe = min(kBwX, W - x0), ye = min(kBwY, H - y0), rows = min(kBwD, D - d0) * kBwY;
        for (int row = part; row < rows; row += parts) {
          if (row % kBwY >= ye) continue;
          const float *z0 = s_dz + o * kBwDz + row * kBwX;
          const float *v = s_in + c * kBwIn + (row / kBwY * (kBwY + 2) + row % kBwY) * kBwRow;
#pragma unroll 1
          for (int x = 0; x < xe; x += 4) {
            const float4 ga = *reinterpret_cast<const float4 *>(z0 + x);
            const float4 gb = *reinterpret_cast<const float4 *>(z0 + kBwDz + x);
            const float g0[4] = {ga.x, ga.y, ga.z, ga.w}, g1[4] = {gb.x, gb.y, gb.z, gb.w};
#pragma unroll
            for (int r = 0; r < 9; ++r) {  // tap rows (dz, dy)
              const float *w = v + (r / 3 * (kBwY + 2) + r % 3) * kBwRow + x;
              const float4 a = *reinterpret_cast<const float4 *>(w);
              const float2 b = *reinterpret_cast<const float2 *>(w + 4);
              const float e[6] = {a.x, a.y, a.z, a.w, b.x, b.y};
#pragma unroll
              for (int k = 0; k < 3; ++k)
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                  acc0[3 * r + k] = __fmaf_rn(g0[i], e[i + k], acc0[3 * r + k]);
                  acc1[3 * r + k] = __fmaf_rn(g1[i], e[i + k], acc1[3 * r + k]);
                }
            }
          }
        }
      }
    }
  }
  if (!any || !active) return;
  float *out = dw + ((static_cast<long long>(f) * co + o) * ci + c) * kTaps;
  unsigned long long bad = 0;  // bit t: acc0[t], bit 32 + t: acc1[t]
#pragma unroll
  for (int t = 0; t < 27; ++t) {
    if (not_finite(acc0[t]))
      bad |= 1ull << t;
    else
      atomicAdd(out + t, acc0[t]);
    if (o + 1 >= co) continue;
    if (not_finite(acc1[t]))
      bad |= 1ull << (32 + t);
    else
      atomicAdd(out + static_cast<long long>(ci) * kTaps + t, acc1[t]);
  }
  for (; bad; bad &= bad - 1) {
    const int b = __ffsll(static_cast<long long>(bad)) - 1, t = b & 31, k = b >> 5;
    float sum = 0.0f;
    count = 0;
    for (int s = 0; s < n; ++s) {  // this thread's rows of this CTA's tiles
      if ((face ? face[s] : 0) != f) continue;
      const float *v = in + (static_cast<long long>(s) * ci + c) * P;
      const float *g = dz + (static_cast<long long>(s) * co + o + k) * P;
      int q = static_cast<int>((blockIdx.x + gridDim.x - count % gridDim.x) % gridDim.x);
      for (; q < tiles; q += gridDim.x) {
        const int x0 = q % tx * kBwX, y0 = q / tx % ty * kBwY, d0 = q / (tx * ty) * kBwD;
        for (int row = part; row < kBwD * kBwY; row += parts) {
          const int d = d0 + row / kBwY, y = y0 + row % kBwY;
          if (d < D && y < H) sum = bw_checked(v, g, t, d, d + 1, y, y + 1, x0, min(x0 + kBwX, W), D, H, W, sum);
        }
      }
      count += tiles;
    }
    atomicAdd(out + static_cast<long long>(k) * ci * kTaps + t, sum);
  }
}

// The same with one CTA per sample, for many samples whose planes fit in shared
// memory: a thread (one input channel, two output channels, 27 taps) walks all
// of the sample's voxels in the order (d, y, x), so every sum of a sample is the
// one sequential chain it has always been.  The input planes d - 1, d, d + 1 and
// dz's plane d are resident, and with PRE the next ones arrive by cp.async while
// d is computed.  Two or three threads share the taps of a pair of outputs,
// which gives every scheduler two warps; 216 FMAs per 4 columns and pair
// against 22 to 24 shared loads.  B200, 128 samples of 8 x 16 x 16 (three layers):
// 167 + 180 + 147 us against 435 us in all for the tiles above, which below about
// 64 samples fill the chip better; taken from there on because a training step
// then differs from the one before by the order of the atomic adds alone.
struct BsGeom {
  int pitch, in_ch, dz_ch;  // input row, floats of a channel's plane (in, dz)
  int bytes(int ci, int co, bool pre) const {
    return 4 * ((pre ? 4 : 3) * ci * in_ch + (pre ? 2 : 1) * 2 * ((co + 1) / 2) * dz_ch);
  }
};
// channels start 4 (mod 8) floats apart modulo the 32 banks
__host__ __device__ inline BsGeom bs_geom(int H, int W) {
  const int wg = (W + 3) / 4 * 4;
  BsGeom g;
  g.pitch = wg + 4;
  g.in_ch = (H + 2) * g.pitch;
  g.in_ch += (12 - g.in_ch % 8) % 8;
  g.dz_ch = H * wg;
  g.dz_ch += (12 - g.dz_ch % 8) % 8;
  return g;
}
// The nine tap rows (dz, dy) are split between three groups of threads (0-2,
// 3-5, 6-8), or between two (0-4, 5-8) where three groups of ci * co / 2 threads
// would not fit in kBsThreads.
constexpr int kBsThreads = 288;

__device__ __forceinline__ void cp_async4(float *dst, const float *src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(
                   static_cast<uint32_t>(__cvta_generic_to_shared(dst))),
               "l"(src)
               : "memory");
}

// One plane of a thread's sums for the tap rows (dz, dy) R0 .. R1 - 1.
template <int R0, int R1>
__device__ __forceinline__ void bs_plane(const float *z0, const float *z1, const float *const v[3], int H,
                                         int wg, int pitch, float acc0[15], float acc1[15]) {
  for (int y = 0; y < H; ++y) {
#pragma unroll 1
    for (int x = 0; x < wg; x += 4) {
      const float4 ga = *reinterpret_cast<const float4 *>(z0 + y * wg + x);
      const float4 gb = *reinterpret_cast<const float4 *>(z1 + y * wg + x);
      const float g0[4] = {ga.x, ga.y, ga.z, ga.w}, g1[4] = {gb.x, gb.y, gb.z, gb.w};
#pragma unroll
      for (int r = R0; r < R1; ++r) {
        const float *w = v[r / 3] + (y + r % 3) * pitch + x;
        const float4 a = *reinterpret_cast<const float4 *>(w);
        const float2 b = *reinterpret_cast<const float2 *>(w + 4);
        const float e[6] = {a.x, a.y, a.z, a.w, b.x, b.y};
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
          for (int k = 0; k < 3; ++k) {
            acc0[3 * (r - R0) + k] = __fmaf_rn(g0[i], e[i + k], acc0[3 * (r - R0) + k]);
            acc1[3 * (r - R0) + k] = __fmaf_rn(g1[i], e[i + k], acc1[3 * (r - R0) + k]);
          }
      }
    }
  }
}

template <bool PRE>
__global__ void __launch_bounds__(kBsThreads, 1)
    k_conv_bwd_weight_seq(const float *in, const float *dz, const int *face, float *dw, int ci, int co,
                          int D, int H, int W, int nface) {
  extern __shared__ __align__(16) float s_t[];
  const int s = blockIdx.x, f = face ? face[s] : 0;
  if (f < 0 || f >= nface) return;
  constexpr int NI = PRE ? 4 : 3, NZ = PRE ? 2 : 1;
  const BsGeom G = bs_geom(H, W);
  const int tid = threadIdx.x, wg = (W + 3) / 4 * 4, co2 = (co + 1) / 2;
  const int span = (ci * co2 + 31) / 32 * 32;  // threads of a group: whole warps
  const bool three = 3 * span <= kBsThreads;
  const int grp = tid / span, c = (tid % span) % ci, o = 2 * ((tid % span) / ci);
  const bool active = o < co;
  const int nin = ci * G.in_ch, ndz = 2 * co2 * G.dz_ch;
  float *const s_in = s_t, *const s_dz = s_t + NI * nin;
  const long long HW = static_cast<long long>(H) * W, P = HW * D;
  const float *src = in + static_cast<long long>(s) * ci * P, *g = dz + static_cast<long long>(s) * co * P;
  // halos, the columns past W and a missing last channel stay zero
  for (int i = tid; i < NI * nin + NZ * ndz; i += blockDim.x) s_t[i] = 0.0f;
  __syncthreads();
  auto load_in = [&](int d) {  // plane d into its slot (d = D: zeros)
    float *dst = s_in + (d + 1) % NI * nin;
    for (int i = tid >> 4; i < ci * H; i += blockDim.x / 16) {
      const int ch = i / H, y = i % H;
      for (int x = tid & 15; x < W; x += 16) {
        float *q = dst + ch * G.in_ch + (y + 1) * G.pitch + 1 + x;
        if (d < D)
          cp_async4(q, src + ch * P + d * HW + static_cast<long long>(y) * W + x);
        else
          *q = 0.0f;
      }
    }
  };
  auto load_dz = [&](int d) {
    float *dst = s_dz + d % NZ * ndz;
    for (int i = tid >> 4; i < co * H; i += blockDim.x / 16) {
      const int ch = i / H, y = i % H;
      for (int x = tid & 15; x < W; x += 16)
        cp_async4(dst + ch * G.dz_ch + y * wg + x, g + ch * P + d * HW + static_cast<long long>(y) * W + x);
    }
  };
  auto arrived = [&]() {
    asm volatile("cp.async.wait_all;" ::: "memory");
    __syncthreads();
  };
  float acc0[15], acc1[15];
#pragma unroll
  for (int t = 0; t < 15; ++t) acc0[t] = acc1[t] = 0.0f;
  load_in(0);
  load_in(1);
  load_dz(0);
  arrived();
  for (int d = 0; d < D; ++d) {
    if (PRE && d + 1 < D) {
      load_in(d + 2);
      load_dz(d + 1);
    }
    if (active) {
      const float *z0 = s_dz + d % NZ * ndz + o * G.dz_ch;
      const float *v[3];
#pragma unroll
      for (int k = 0; k < 3; ++k) v[k] = s_in + (d + k) % NI * nin + c * G.in_ch;
      const float *z1 = z0 + G.dz_ch;
      if (three) {
        if (grp == 0) bs_plane<0, 3>(z0, z1, v, H, wg, G.pitch, acc0, acc1);
        if (grp == 1) bs_plane<3, 6>(z0, z1, v, H, wg, G.pitch, acc0, acc1);
        if (grp == 2) bs_plane<6, 9>(z0, z1, v, H, wg, G.pitch, acc0, acc1);
      } else {
        if (grp == 0) bs_plane<0, 5>(z0, z1, v, H, wg, G.pitch, acc0, acc1);
        if (grp == 1) bs_plane<5, 9>(z0, z1, v, H, wg, G.pitch, acc0, acc1);
      }
    }
    if (PRE) {
      arrived();
    } else if (d + 1 < D) {
      __syncthreads();  // plane d - 1's slot and dz are free
      load_in(d + 2);
      load_dz(d + 1);
      arrived();
    }
  }
  if (!active) return;
  const int t0 = grp * (three ? 9 : 15), nt = min(three ? 9 : 15, kTaps - t0);
  float *out = dw + ((static_cast<long long>(f) * co + o) * ci + c) * kTaps + t0;
  unsigned bad = 0;  // bit t: acc0[t], bit 16 + t: acc1[t]
#pragma unroll
  for (int t = 0; t < 15; ++t) {
    if (t >= nt) break;
    if (not_finite(acc0[t]))
      bad |= 1u << t;
    else
      atomicAdd(out + t, acc0[t]);
    if (o + 1 >= co) continue;
    if (not_finite(acc1[t]))
      bad |= 1u << (16 + t);
    else
      atomicAdd(out + static_cast<long long>(ci) * kTaps + t, acc1[t]);
  }
  for (; bad; bad &= bad - 1) {
    const int b = __ffs(bad) - 1, t = b & 15, k = b >> 4;
    atomicAdd(out + static_cast<long long>(k) * ci * kTaps + t,
              bw_checked(src + c * P, g + (o + k) * P, t0 + t, 0, D, 0, H, 0, W, D, H, W, 0.0f));
  }
}

__global__ void k_gelu_bwd(const float *da, const float *z, float *dz, long long m) {
  const long long i = static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x;
  if (i < m) dz[i] = da[i] * gelu_grad(z[i]);
}

// loss += sum (y - t)^2 / m;  dy = 2 (y - t) / m.  A grid stride over a few
// CTAs per SM: one atomic per CTA on the loss, where one per 256 values queued
// up on its address (1.6 M values: 15 us with 6144 of them).
__global__ void k_mse(const float *y, const float *t, float *dy, float *loss, long long m) {
  __shared__ float s_sum[256];
  float acc = 0.0f;
  for (long long i = static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x; i < m;
       i += static_cast<long long>(gridDim.x) * blockDim.x) {
    const float d = y[i] - t[i];
    dy[i] = 2.0f * d / static_cast<float>(m);
    acc += d * d;
  }
  s_sum[threadIdx.x] = acc;
  __syncthreads();
  for (int k = blockDim.x / 2; k > 0; k >>= 1) {
    if (threadIdx.x < k) s_sum[threadIdx.x] += s_sum[threadIdx.x + k];
    __syncthreads();
  }
  if (threadIdx.x == 0) atomicAdd(loss, s_sum[0] / static_cast<float>(m));
}

// Adam (Kingma & Ba) on FP32 master weights; the bfloat16 copy is what the
// forward pass reads.
__global__ void k_adam(float *w, __nv_bfloat16 *wb, const float *g, float *m1, float *m2, long long n,
                       float lr, float b1, float b2, float eps, float c1, float c2) {
  const long long i = static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const float gi = g[i];
  const float a = b1 * m1[i] + (1.0f - b1) * gi;
  const float b = b2 * m2[i] + (1.0f - b2) * gi * gi;
  m1[i] = a;
  m2[i] = b;
  const float wi = w[i] - lr * (a / c1) / (sqrtf(b / c2) + eps);
  w[i] = wi;
  wb[i] = __float2bfloat16_rn(wi);
}

// ---- band gather / scatter on a grid's state --------------------------------

// X[f][10][8][H][W]: 6 fields scaled by gain (E by ge, H by gh), then the 4
// psi of the face's normal axis (terms of E differences by ge, of H by gh).
// One launch per axis covers its two faces.
template <int AX>
__global__ void __launch_bounds__(256) k_band_gather(BandGrid g, float *X, int H, int W, float ge,
                                                     float gh) {
  using T = BandTile<AX>;
  __shared__ float s[kBandIn][T::TO][T::TA][33];
  const int side = blockIdx.z / T::kZ, sub = blockIdx.z % T::kZ, f = 2 * AX + side;
  const int v0 = blockIdx.x * 32;
  const long long P = static_cast<long long>(kBandDepth) * H * W;
  const BandPsi &ps = g.psi[AX];
#pragma unroll
  for (int j = 0; j < T::kElems / 256; ++j) {  // grid side: a fastest
    const int e = threadIdx.x + 256 * j, al = e % T::TA, vl = (e / T::TA) % 32, ol = e / (T::TA * 32);
    int d, u;
    band_du<AX>(al, ol, blockIdx.y, sub, d, u);
    const int v = v0 + vl;
    if (d < kBandDepth && u < H && v < W) {
      int x, y, z;
      band_cell(g, f, d, u, v, x, y, z);
      const long long cell = (static_cast<long long>(z) * g.ny + y) * g.nx + x;
#pragma unroll
      for (int c = 0; c < 6; ++c) s[c][ol][al][vl] = g.fields[c * g.N + cell] * (c < 3 ? ge : gh);
      const long long k = psi_index(g, AX, x, y, z);
#pragma unroll
      for (int c = 0; c < 4; ++c)
        s[6 + c][ol][al][vl] = k >= 0 ? ps.p[c * ps.cells + k] * (c < 2 ? ge : gh) : 0.0f;
    }
  }
  __syncthreads();
#pragma unroll
  for (int j = 0; j < T::kElems / 256; ++j) {  // band side: v fastest
    const int e = threadIdx.x + 256 * j, vl = e % 32, al = (e / 32) % T::TA, ol = e / (32 * T::TA);
    int d, u;
    band_du<AX>(al, ol, blockIdx.y, sub, d, u);
    const int v = v0 + vl;
    if (d < kBandDepth && u < H && v < W) {
      float *out = X + static_cast<long long>(f) * kBandIn * P + (static_cast<long long>(d) * H + u) * W + v;
#pragma unroll
      for (int c = 0; c < kBandIn; ++c) out[c * P] = s[c][ol][al][vl];
    }
  }
}

// fields += Y / gain over the bands of faces f0 .. f0 + nf - 1 (both faces of
// axis AX in one launch when their bands are disjoint).  The axes go in
// order, so a cell in two bands gets both corrections, edges first by the
// lower face index.
template <int AX>
__global__ void __launch_bounds__(256) k_band_scatter_add(BandGrid g, const float *Y, int H, int W,
                                                          float ge, float gh, int f0) {
  using T = BandTile<AX>;
  __shared__ float s[6][T::TO][T::TA][33];
  const int f = f0 + blockIdx.z / T::kZ, sub = blockIdx.z % T::kZ, v0 = blockIdx.x * 32;
  const long long P = static_cast<long long>(kBandDepth) * H * W;
#pragma unroll
  for (int j = 0; j < T::kElems / 256; ++j) {  // band side: v fastest
    const int e = threadIdx.x + 256 * j, vl = e % 32, al = (e / 32) % T::TA, ol = e / (32 * T::TA);
    int d, u;
    band_du<AX>(al, ol, blockIdx.y, sub, d, u);
    const int v = v0 + vl;
    if (d < kBandDepth && u < H && v < W) {
      const float *in = Y + static_cast<long long>(f) * 6 * P + (static_cast<long long>(d) * H + u) * W + v;
#pragma unroll
      for (int c = 0; c < 6; ++c) s[c][ol][al][vl] = in[c * P];
    }
  }
  __syncthreads();
#pragma unroll
  for (int j = 0; j < T::kElems / 256; ++j) {  // grid side: a fastest
    const int e = threadIdx.x + 256 * j, al = e % T::TA, vl = (e / T::TA) % 32, ol = e / (T::TA * 32);
    int d, u;
    band_du<AX>(al, ol, blockIdx.y, sub, d, u);
    const int v = v0 + vl;
    if (d < kBandDepth && u < H && v < W) {
      int x, y, z;
      band_cell(g, f, d, u, v, x, y, z);
      const long long cell = (static_cast<long long>(z) * g.ny + y) * g.nx + x;
#pragma unroll
      for (int c = 0; c < 6; ++c) g.fields[c * g.N + cell] += s[c][ol][al][vl] / (c < 3 ? ge : gh);
    }
  }
}

// Student state (nx, ny, nz) = teacher state at offset `off` on every axis:
// the six fields, and on each axis the student's psi slab from the teacher's
// psi at the same physical cells.
__global__ void k_restrict(BandGrid t, BandGrid s, int off) {
  const long long i = static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x;
  if (i >= s.N) return;
  const int x = static_cast<int>(i % s.nx), y = static_cast<int>((i / s.nx) % s.ny), z = static_cast<int>(i / (static_cast<long long>(s.nx) * s.ny));
  const int X = x + off, Y = y + off, Z = z + off;
  const long long ti = (static_cast<long long>(Z) * t.ny + Y) * t.nx + X;
  for (int c = 0; c < 6; ++c) s.fields[c * s.N + i] = t.fields[c * t.N + ti];
  for (int ax = 0; ax < 3; ++ax) {
    const long long ks = psi_index(s, ax, x, y, z);
    if (ks < 0) continue;
    const long long kt = psi_index(t, ax, X, Y, Z);
    for (int c = 0; c < 4; ++c)
      s.psi[ax].p[c * s.psi[ax].cells + ks] = kt >= 0 ? t.psi[ax].p[c * t.psi[ax].cells + kt] : 0.0f;
  }
}

// s[f] = RMS of the E channels (0..2) of face f's band tensor (a tiny floor
// keeps an all-zero band at zero after scaling).
__global__ void k_face_rms(const float *X, int C, long long P, float *s) {
  __shared__ float s_sum[256];
  const int f = blockIdx.x;
  const float *x = X + static_cast<long long>(f) * C * P;
  float acc = 0.0f;
  for (long long i = threadIdx.x; i < 3 * P; i += blockDim.x) acc += x[i] * x[i];
  s_sum[threadIdx.x] = acc;
  __syncthreads();
  for (int k = blockDim.x / 2; k > 0; k >>= 1) {
    if (threadIdx.x < k) s_sum[threadIdx.x] += s_sum[threadIdx.x + k];
    __syncthreads();
  }
  if (threadIdx.x == 0) s[f] = sqrtf(s_sum[0] / static_cast<float>(3 * P)) + 1e-30f;
}

// Energy guard of a face's correction Y (field units times the gains) on its
// band fields F = X * s[f] (X normalised, channels 0-5 the fields): with
// a = <F, Y> and b = <Y, Y> over the six field channels, the band energy
// changes by 2a + b; if that is positive, lam[f] = clamp(-2a / b, 0, 1) is the
// largest factor that keeps it from growing, else lam[f] = 1.
__global__ void k_face_guard(const float *X, int C, const float *Y, long long P, const float *s,
                             float *lam) {
  __shared__ float s_a[256], s_b[256];
  const int f = blockIdx.x;
  const float *x = X + static_cast<long long>(f) * C * P;
  const float *y = Y + static_cast<long long>(f) * 6 * P;
  float a = 0.0f, b = 0.0f;
  for (long long i = threadIdx.x; i < 6 * P; i += blockDim.x) {
    a += x[i] * y[i];
    b += y[i] * y[i];
  }
  s_a[threadIdx.x] = a;
  s_b[threadIdx.x] = b;
  __syncthreads();
  for (int k = blockDim.x / 2; k > 0; k >>= 1) {
    if (threadIdx.x < k) {
      s_a[threadIdx.x] += s_a[threadIdx.x + k];
      s_b[threadIdx.x] += s_b[threadIdx.x + k];
    }
    __syncthreads();
  }
  if (threadIdx.x == 0) {
    const float aa = s_a[0] * s[f], bb = s_b[0];
    float l = 1.0f;
    if (2.0f * aa + bb > 0.0f) l = (aa < 0.0f && bb > 0.0f) ? fminf(1.0f, -2.0f * aa / bb) : 0.0f;
    lam[f] = l;
  }
}

// X[f][c][p] *= s[f] (or / s[f])
__global__ void k_face_scale(float *X, int C, long long P, const float *s, int divide) {
  const long long i = static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x;
  const int f = blockIdx.y;
  if (i >= C * P) return;
  const float m = divide ? 1.0f / s[f] : s[f];
  X[static_cast<long long>(f) * C * P + i] *= m;
}

inline unsigned blocks_for(long long n, int t) { return static_cast<unsigned>((n + t - 1) / t); }

}  // namespace

// Which kernels run the forward and input-gradient convolutions: the
// tensor-core implicit GEMMs (wf_conv_tc.cu, the default) or the CUDA-core
// kernels above.
static int g_nn_tensor_cores = 1;
void nn_set_tensor_cores(int on) { g_nn_tensor_cores = on != 0; }
int nn_tensor_cores() { return g_nn_tensor_cores; }

int nn_conv_fwd(const float *in, const void *w_bf16, const int *face, float *z, float *a, int n,
                int ci, int co, int D, int H, int W, int act, void *stream) {
  if (ci > kMaxC || co > kMaxC || ci < 1 || co < 1 || n < 1) return cudaErrorInvalidValue;
  if (g_nn_tensor_cores) return nn_conv_fwd_tc(in, w_bf16, face, z, a, n, ci, co, D, H, W, act, stream);
  const long long P = static_cast<long long>(D) * H * W;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  const __nv_bfloat16 *wb = static_cast<const __nv_bfloat16 *>(w_bf16);
  if (co == 16 || co == 6) {  // the network's layers: the blocked kernel
    const long long quads = static_cast<long long>(D) * H * ((W + 3) / 4);
    dim3 grid(blocks_for(quads, 128), n);
    const size_t sm = sizeof(float) * ci * kTaps * (co == 16 ? 16 : 8);
    if (co == 16)
      k_conv_fwd4<16><<<grid, 128, sm, st>>>(in, wb, face, z, a, n, ci, D, H, W, act);
    else
      k_conv_fwd4<6><<<grid, 128, sm, st>>>(in, wb, face, z, a, n, ci, D, H, W, act);
    return cudaGetLastError();
  }
  dim3 grid(blocks_for(P, 128), n);
  k_conv_fwd<<<grid, 128, sizeof(float) * co * ci * kTaps, st>>>(in, wb, face, z, a, n, ci, co, D,
                                                                  H, W, act);
  return cudaGetLastError();
}

int nn_conv_bwd_data(const float *dz, const void *w_bf16, const int *face, float *din, int n,
                     int ci, int co, int D, int H, int W, void *stream) {
  if (ci > kMaxC || co > kMaxC || ci < 1 || co < 1 || n < 1) return cudaErrorInvalidValue;
  if (g_nn_tensor_cores) return nn_conv_bwd_data_tc(dz, w_bf16, face, din, n, ci, co, D, H, W, stream);
  const long long P = static_cast<long long>(D) * H * W;
  dim3 grid(blocks_for(P, 128), n);
  k_conv_bwd_data<<<grid, 128, sizeof(float) * co * ci * kTaps, static_cast<cudaStream_t>(stream)>>>(
      dz, static_cast<const __nv_bfloat16 *>(w_bf16), face, din, n, ci, co, D, H, W);
  return cudaGetLastError();
}

int nn_conv_bwd_weight(const float *in, const float *dz, const int *face, float *dw, int n, int ci,
                       int co, int D, int H, int W, int nface, void *stream) {
  if (ci > kMaxC || co > kMaxC || nface > 8 || n < 1) return cudaErrorInvalidValue;
  if (ci < 1 || co < 1) return cudaErrorInvalidConfiguration;  // as an empty launch grid
  if (nface < 1 || D < 1 || H < 1 || W < 1) return cudaSuccess;  // nothing to add
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  if (n < 64 && static_cast<long long>(D) * H * W <= kBwFewVoxels) {
    const dim3 grid(blocks_for(co * ci * kTaps, 128), std::min(n, 64));
    k_conv_bwd_weight_few<<<grid, 128, 0, st>>>(in, dz, face, dw, n, ci, co, D, H, W, nface);
    return cudaGetLastError();
  }
  // one CTA per sample where there are enough samples and the planes fit
  const BsGeom G = bs_geom(H, W);
  constexpr int kSmemMax = 227 * 1024;
  if (n >= 64 && H <= 256 && W <= 256 && G.bytes(ci, co, false) <= kSmemMax) {
    const bool pre = G.bytes(ci, co, true) <= kSmemMax;
    auto fn = pre ? k_conv_bwd_weight_seq<true> : k_conv_bwd_weight_seq<false>;
    cudaError_t e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmemMax);
    if (e != cudaSuccess) return e;
    const int span = (ci * ((co + 1) / 2) + 31) / 32 * 32;
    fn<<<n, 3 * span <= kBsThreads ? 3 * span : 2 * span, G.bytes(ci, co, pre), st>>>(in, dz, face, dw, ci, co, D, H, W, nface);
    return cudaGetLastError();
  }
  cudaError_t e = cudaFuncSetAttribute(k_conv_bwd_weight, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       kBwSmem);
  if (e != cudaSuccess) return e;
  int dev = 0, nsm = 0;
  e = cudaGetDevice(&dev);
  if (e == cudaSuccess) e = cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
  if (e != cudaSuccess) return e;
  // two CTAs per SM over the faces, never more than there are tiles
  const long long tiles = static_cast<long long>(n) * ((W + kBwX - 1) / kBwX) *
                          ((H + kBwY - 1) / kBwY) * ((D + kBwD - 1) / kBwD);
  const long long want = std::max(1, 2 * nsm / nface);
  dim3 grid(static_cast<unsigned>(std::min(want, tiles)), nface);
  k_conv_bwd_weight<<<grid, kBwThreads, kBwSmem, st>>>(in, dz, face, dw, n, ci, co, D, H, W);
  return cudaGetLastError();
}

int nn_gelu_bwd(const float *da, const float *z, float *dz, long long m, void *stream) {
  k_gelu_bwd<<<blocks_for(m, 256), 256, 0, static_cast<cudaStream_t>(stream)>>>(da, z, dz, m);
  return cudaGetLastError();
}

int nn_mse(const float *y, const float *t, float *dy, float *loss, long long m, void *stream) {
  if (m < 1) return cudaErrorInvalidConfiguration;  // as an empty launch grid
  const unsigned blocks = std::min(blocks_for(m, 256), 592u);
  k_mse<<<blocks, 256, 0, static_cast<cudaStream_t>(stream)>>>(y, t, dy, loss, m);
  return cudaGetLastError();
}

int nn_adam(float *w, void *w_bf16, const float *g, float *m1, float *m2, long long n, float lr,
            float b1, float b2, float eps, int t, void *stream) {
  const float c1 = 1.0f - powf(b1, static_cast<float>(t)), c2 = 1.0f - powf(b2, static_cast<float>(t));
  k_adam<<<blocks_for(n, 256), 256, 0, static_cast<cudaStream_t>(stream)>>>(
      w, static_cast<__nv_bfloat16 *>(w_bf16), g, m1, m2, n, lr, b1, b2, eps, c1, c2);
  return cudaGetLastError();
}

int band_gather(const BandGrid &g, float *X, int H, int W, float ge, float gh, void *stream) {
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  const unsigned bx = blocks_for(W, 32);
  k_band_gather<0><<<dim3(bx, blocks_for(H, BandTile<0>::TO), 2 * BandTile<0>::kZ), 256, 0, st>>>(
      g, X, H, W, ge, gh);
  k_band_gather<1><<<dim3(bx, blocks_for(H, 32), 2 * BandTile<1>::kZ), 256, 0, st>>>(g, X, H, W, ge, gh);
  k_band_gather<2><<<dim3(bx, blocks_for(H, 32), 2 * BandTile<2>::kZ), 256, 0, st>>>(g, X, H, W, ge, gh);
  return cudaGetLastError();
}

int band_scatter_add(const BandGrid &g, const float *Y, int H, int W, float ge, float gh,
                     void *stream) {
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  const unsigned bx = blocks_for(W, 32);
  const int extent[3] = {g.nx, g.ny, g.nz};
  for (int ax = 0; ax < 3; ++ax) {
    // the two faces' bands are disjoint when the axis holds two band depths
    const int nf = extent[ax] >= 2 * kBandDepth ? 2 : 1;
    for (int f = 2 * ax; f < 2 * ax + 2; f += nf) {
      if (ax == 0)
        k_band_scatter_add<0><<<dim3(bx, blocks_for(H, BandTile<0>::TO), nf * BandTile<0>::kZ), 256, 0,
                                st>>>(g, Y, H, W, ge, gh, f);
      else if (ax == 1)
        k_band_scatter_add<1><<<dim3(bx, blocks_for(H, 32), nf * BandTile<1>::kZ), 256, 0, st>>>(
            g, Y, H, W, ge, gh, f);
      else
        k_band_scatter_add<2><<<dim3(bx, blocks_for(H, 32), nf * BandTile<2>::kZ), 256, 0, st>>>(
            g, Y, H, W, ge, gh, f);
    }
  }
  return cudaGetLastError();
}

int face_rms(const float *X, int C, long long P, float *s, void *stream) {
  k_face_rms<<<6, 256, 0, static_cast<cudaStream_t>(stream)>>>(X, C, P, s);
  return cudaGetLastError();
}

int face_guard(const float *X, int C, const float *Y, long long P, const float *s, float *lam,
               void *stream) {
  k_face_guard<<<6, 256, 0, static_cast<cudaStream_t>(stream)>>>(X, C, Y, P, s, lam);
  return cudaGetLastError();
}

int face_scale(float *X, int C, long long P, const float *s, int divide, void *stream) {
  k_face_scale<<<dim3(blocks_for(C * P, 256), 6), 256, 0, static_cast<cudaStream_t>(stream)>>>(X, C, P, s, divide);
  return cudaGetLastError();
}

int band_restrict(const BandGrid &teacher, const BandGrid &student, int off, void *stream) {
  k_restrict<<<blocks_for(student.N, 256), 256, 0, static_cast<cudaStream_t>(stream)>>>(teacher, student, off);
  return cudaGetLastError();
}

}  // namespace wf
