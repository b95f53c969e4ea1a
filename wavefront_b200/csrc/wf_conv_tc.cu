// wf_conv_tc.cu -- the closure network's 3x3x3 convolutions on the sm_100a
// tensor cores (tcgen05.mma, accumulators in tensor memory), as implicit
// GEMMs on FP32 tensors: the training path and the closure's generic one.
//
// Numerics.  The weights are bfloat16 (exact operands).  An FP32 activation
// a is split into three bfloat16 parts, a1 = bf16(a), a2 = bf16(a - a1),
// a3 = bf16(a - a1 - a2) (each difference exact in FP32), and every part is
// multiplied by the weight: the operand keeps 24 significant bits, like FP32
// itself (two parts would keep 16, a relative error up to 2^-16), every
// product is exact, and the tensor core accumulates in FP32.  Results agree
// with the FP32 CUDA-core kernels to about 1e-6 relative, not bit for bit
// (the summation order differs), and with the in-step closure's
// (wf_closure_fast.cu) operand by operand: the same sums in the same order.
//
// One MMA of M 128 x N 48 x K 16 multiplies 128 consecutive staged voxels of an
// input plane, shifted by a tap (dy, dx), with that tap's weights for dz = +1,
// 0, -1 stacked along N: it adds to output planes z - 1, z, z + 1.  An M 128 x
// K 16 MMA takes the same 48 cycles for every N up to 64.  Per output the taps
// are summed in the order (dz, dy, dx, part).
//
// Data layout in shared memory (no swizzle, K-major canonical layout: core
// matrices of 8 rows x 16 bytes):
//   A  [plane][part 1..3][channel half][guard, rows of `pitch` voxels, guard] x
//      8 channels (16 bytes a voxel): up to 6 input planes around the CTA's 4
//      output planes.  Rows of at most 31 columns are staged whole, with one
//      zero column after them that is also the halo before the next row
//      (pitch W + 1, 128 / pitch output rows a tile); wider ones as 30 columns
//      and both halos (pitch 32, 4 rows).  One M tile is 128 consecutive voxels,
//      so a tap only moves its start address by dy * pitch + dx voxels.
//   B  [dy, dx][channel half][n = 16 j + co][8 input channels], row block j
//      holding dz = 1 - j
// Tensor memory: 8 planes x 16 FP32 columns, the CTA's 4 output planes in the
// middle (the outer ones take the products of out-of-tile taps and are never
// read).
//
// One thread issues all MMAs of the CTA and commits them to an mbarrier;
// the wait is bounded (a timeout is counted, the epilogue is skipped and the
// tensor memory is still freed).
//
// Measured on B200 (128 samples of 8 x 16 x 16, 16 -> 16 channels): 130 us with
// one N 16 MMA per tap and part over 2 planes x 4 rows x 32 columns, half of
// them padding here; 50 us now, two CTAs an SM whose load, MMA and epilogue
// phases overlap.  (N 144 with the dx taps stacked too took 25 us, but sums in
// another order: training results then differ from before by more than the
// FP32 rounding of one order.)
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include "wf_band.cuh"
#include "wf_closure.h"
#include "wf_internal.cuh"

namespace wf {

namespace {

constexpr int kTcD = 4;                  // output planes per CTA
constexpr int kTcN = 48;                 // MMA N: three planes x 16 outputs
constexpr int kTcWHalf = kTcN * 16;      // one K half of a (dy, dx) block of weights
constexpr int kTcWBytes = 9 * 2 * kTcWHalf;
constexpr int kTcThreads = 256;          // 8 warps: two per TMEM lane quarter
constexpr int kTcCols = 16 * (kTcD + 4);  // tensor-memory columns: 128
constexpr int kTcZero = 4096;            // zeros: A and B of the clearing MMA (128 rows each)
constexpr int kTcMaxRow = 31;            // rows staged whole up to this width
static_assert(kTcCols == 128, "a power of two, and the clearing MMA's N");

// Tile geometry of a width: pitch, output columns and rows, the bytes of one
// [part][half] array (2 halo rows, 128 voxels and 2 guards) and the total.
struct TcGeom {
  int pitch, outc, rows, arr, bytes;
};
__host__ __device__ inline TcGeom tc_geom(int W) {
  TcGeom g;
  g.pitch = W <= kTcMaxRow ? W + 1 : 32;
  g.outc = W <= kTcMaxRow ? W : 30;
  g.rows = 128 / g.pitch;
  g.arr = (2 * g.pitch + 128 + 2) * 16;
  g.bytes = kTcWBytes + kTcZero + 16 + (kTcD + 2) * 6 * g.arr;
  return g;
}

// The most any width takes: the function's shared-memory limit, always the same
// one, because it belongs to the function on the device and another thread may
// be between its own limit and its launch with another width.
constexpr int kTcMaxBytes = kTcWBytes + kTcZero + 16 + (kTcD + 2) * 6 * (2 * 32 + 128 + 2) * 16;

__device__ unsigned long long g_tc_timeouts;  // bounded-wait expiries (diagnostic)

constexpr float kInvSqrt2f = 0.70710678118654752f;
__device__ __forceinline__ float gelu_f(float z) { return 0.5f * z * (1.0f + erff(z * kInvSqrt2f)); }

// Shared-memory matrix descriptor, no swizzle (sm_100 version 1).
__device__ __forceinline__ uint64_t smem_desc(uint32_t addr, uint32_t lbo, uint32_t sbo) {
  return static_cast<uint64_t>((addr >> 4) & 0x3FFFu) |
         (static_cast<uint64_t>((lbo >> 4) & 0x3FFFu) << 16) |
         (static_cast<uint64_t>((sbo >> 4) & 0x3FFFu) << 32) | (1ull << 46);
}

// kind::f16, BF16 A and B (K-major), FP32 D, M = 128, N = n
__host__ __device__ constexpr uint32_t idesc_n(uint32_t n) {
  return (1u << 4) | (1u << 7) | (1u << 10) | ((n >> 3) << 17) | ((128u >> 4) << 24);
}

// Issued by the lane with `leader` set, in code that the whole warp runs (see
// wf_closure_fast.cu).
__device__ __forceinline__ void umma_bf16(uint32_t d_tmem, uint64_t a, uint64_t b, uint32_t idesc,
                                          uint32_t accum, uint32_t leader) {
  asm volatile(
      "{\n .reg .pred p, q;\n setp.ne.b32 p, %4, 0;\n setp.ne.b32 q, %5, 0;\n"
      " @q tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n}\n" ::"r"(d_tmem),
      "l"(a), "l"(b), "r"(idesc), "r"(accum), "r"(leader));
}

__device__ __forceinline__ void umma_commit(uint32_t bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar)
               : "memory");
}

__device__ __forceinline__ void tc_fence_before() {
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
}
__device__ __forceinline__ void tc_fence_after() {
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
}

__device__ __forceinline__ void tmem_ld16(uint32_t taddr, float v[16]) {
  uint32_t r[16];
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, "
      "%12, %13, %14, %15}, [%16];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]),
        "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]),
        "=r"(r[14]), "=r"(r[15])
      : "r"(taddr));
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
  for (int i = 0; i < 16; ++i) v[i] = __uint_as_float(r[i]);
}

// out[s][co][p] = sum_ci sum_tap W[tap][co][ci] * in[s][ci][p + tap], with
// W from the bfloat16 weights [F][co][ci][27] (forward) or, for the
// gradient with respect to the input, [F][ci][co][27] transposed and with
// the taps flipped (BWD: in = dz with `kin` = co channels, out = ci).
template <bool BWD>
__global__ void __launch_bounds__(kTcThreads, 2)
    k_conv_tc(const float *in, const __nv_bfloat16 *w, const int *face, float *z, float *a,
              int kin, int nout, int D, int H, int W, int ndt, int act) {
  extern __shared__ __align__(128) unsigned char smem[];
  __shared__ uint32_t s_tmem;
  const TcGeom G = tc_geom(W);
  const int tid = threadIdx.x, lane = tid & 31;
  const int warp = __shfl_sync(0xffffffffu, tid >> 5, 0);  // warp-uniform
  const int s = blockIdx.z / ndt, dt = blockIdx.z % ndt;
  const bool whole = W <= kTcMaxRow;
  const int x0 = blockIdx.x * G.outc, y0 = blockIdx.y * G.rows, dp0 = dt * kTcD;
  const int np = min(kTcD, D - dp0);                            // output planes
  const int zlo = max(dp0 - 1, 0), zhi = min(dp0 + np, D - 1);  // input planes
  const int f = face ? face[s] : 0;
  const long long HW = static_cast<long long>(H) * W, P = HW * D;
  unsigned char *const sW = smem, *const sZ = smem + kTcWBytes, *const sA = sZ + kTcZero + 16;
  const uint32_t sbase = smem_u32(smem), bar = sbase + kTcWBytes + kTcZero;
  const uint32_t a_base = bar + 16;

  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                     smem_u32(&s_tmem)),
                 "r"(kTcCols)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  if (tid == 0) {
    mbar_init(bar, 1);
    mbar_fence_init();
  }
  for (int i = tid; i < kTcZero / 16; i += kTcThreads)
    reinterpret_cast<uint4 *>(sZ)[i] = make_uint4(0u, 0u, 0u, 0u);

  // B: the sample's face's weights, zero padded; the contiguous block is
  // copied as it is (16-byte vectors when it allows) into the A region, which
  // is filled only after, and rearranged 16 bytes at a time from there
  {
    __nv_bfloat16 *raw = reinterpret_cast<__nv_bfloat16 *>(sA);
    const int wn = BWD ? kin : nout;   // first index of the stored weights (co)
    const int wk = BWD ? nout : kin;   // second (ci)
    const int nraw = wn * wk * 27;
    const __nv_bfloat16 *wf = w + static_cast<long long>(f) * nraw;
    if ((nraw % 8) == 0 && (reinterpret_cast<uintptr_t>(wf) & 15) == 0) {
      const uint4 *src = reinterpret_cast<const uint4 *>(wf);
      uint4 *dst = reinterpret_cast<uint4 *>(raw);
      for (int i = tid; i < nraw / 8; i += kTcThreads) dst[i] = __ldg(src + i);
    } else {
      for (int i = tid; i < nraw; i += kTcThreads) raw[i] = wf[i];
    }
    __syncthreads();
    uint4 *sb = reinterpret_cast<uint4 *>(sW);
    for (int i = tid; i < kTcWBytes / 16; i += kTcThreads) {
      const int n = i % kTcN, half = i / kTcN & 1, r = i / (2 * kTcN);
      const int o = n % 16, t = (2 - n / 16) * 9 + r;
      uint32_t q[4];
#pragma unroll
      for (int k2 = 0; k2 < 8; k2 += 2) {
        uint32_t v = 0u;
#pragma unroll
        for (int e = 0; e < 2; ++e) {
          const int k = half * 8 + k2 + e;
          if (o < nout && k < kin)
            v |= static_cast<uint32_t>(__bfloat16_as_ushort(BWD ? raw[(k * wk + o) * 27 + (26 - t)]
                                                                : raw[(o * wk + k) * 27 + t]))
                 << (16 * e);
        }
        q[k2 / 2] = v;
      }
      sb[i] = make_uint4(q[0], q[1], q[2], q[3]);
    }
    __syncthreads();  // the raw copy in the A region is consumed
  }
  // A: the input planes as three bfloat16 parts, zero outside the tensor (the
  // guards, the halos, and the voxels an M tile reads past its last row)
  {
    const float *src = in + static_cast<long long>(s) * kin * P;
    const int nv = 2 * G.pitch + 130, nvox = (zhi - zlo + 1) * nv;
    for (int i = tid; i < nvox; i += kTcThreads) {
      const int pl = i / nv, vx = i % nv - 1;  // -1: the guard before row 0
      const int row = vx >= 0 ? vx / G.pitch : -1, c = vx - row * G.pitch;
      const int d = zlo + pl, y = y0 - 1 + row, x = whole ? c : x0 - 1 + c;
      const bool inside = vx >= 0 && row < G.rows + 2 && y >= 0 && y < H && x >= 0 && x < W;
      const long long off = d * HW + static_cast<long long>(y) * W + x;
      float v[16];
#pragma unroll
      for (int c16 = 0; c16 < 16; ++c16)
        v[c16] = (inside && c16 < kin) ? __ldg(src + c16 * P + off) : 0.0f;
      uint4 q[6];
      split16(v, q);
      uint4 *dst = reinterpret_cast<uint4 *>(sA + pl * 6 * G.arr) + vx + 1;
#pragma unroll
      for (int k = 0; k < 6; ++k) dst[k * (G.arr / 16)] = q[k];
    }
  }
  fence_proxy_async();  // the operands above are read by the tensor core (async proxy)
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = __shfl_sync(0xffffffffu, s_tmem, 0);

  if (warp == 0) {
    const uint32_t leader = lane == 0 ? 1u : 0u, zb = sbase + kTcWBytes;
    umma_bf16(tmem, smem_desc(zb, 2048, 128), smem_desc(zb, 2048, 128), idesc_n(kTcCols), 0u, leader);
    const uint64_t ad0 = smem_desc(a_base + 16, G.arr, 128), bd0 = smem_desc(sbase, kTcWHalf, 128);
    const uint64_t part_off = 2 * static_cast<uint64_t>(G.arr / 16);
    for (int zi = zlo; zi <= zhi; ++zi) {
      const uint32_t d = tmem + 16 * (zi - dp0 + 1);  // planes zi - 1, zi, zi + 1
      const uint64_t az = ad0 + static_cast<uint64_t>((zi - zlo) * 6 * (G.arr / 16));
#pragma unroll
      for (int r = 0; r < 9; ++r) {
        // output row 0, shifted by (dy, dx): staged row 1 + dy, a column more or
        // less (pitch 32: the first staged column is x0 - 1 and dropped)
        const uint64_t ar = az + static_cast<uint64_t>(static_cast<long long>((r / 3) * G.pitch + r % 3 - 1));
        const uint64_t bd = bd0 + static_cast<uint64_t>(r * 2 * kTcWHalf / 16);
#pragma unroll
        for (int part = 0; part < 3; ++part)
          umma_bf16(d, ar + part * part_off, bd, idesc_n(kTcN), 1u, leader);
      }
    }
    if (lane == 0) umma_commit(bar);
    __syncwarp();
  }
  const bool done = mbar_wait(bar, 0);
  tc_fence_after();
  if (!done) {
    if (tid == 0) atomicAdd(&g_tc_timeouts, 1ull);
  } else {
    // epilogue: warp w reads tensor-memory lanes 32 (w % 4) .. + 31 of every
    // second plane from w / 4; lane m is staged voxel m of the output rows
    const int m = 32 * (warp & 3) + lane, row = m / G.pitch, c = m % G.pitch;
    const int y = y0 + row, x = whole ? c : x0 - 1 + c;
    const bool keep = row < G.rows && y < H && x < W && (whole || (c >= 1 && c <= G.outc));
    for (int p = warp >> 2; p < np; p += kTcThreads / 128) {
      float v[16];
      tmem_ld16(tmem + (static_cast<uint32_t>((warp & 3) * 32) << 16) + 16 * (p + 2), v);
      if (keep) {
        const long long q = (dp0 + p) * HW + static_cast<long long>(y) * W + x;
#pragma unroll
        for (int o = 0; o < 16; ++o) {
          if (o >= nout) break;
          const long long k = (static_cast<long long>(s) * nout + o) * P + q;
          if (z) z[k] = v[o];
          a[k] = act ? gelu_f(v[o]) : v[o];
        }
      }
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 0) {
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(kTcCols)
                 : "memory");
  }
}

template <bool BWD>
int launch_tc(const float *in, const void *w, const int *face, float *z, float *a, int n, int kin,
              int nout, int D, int H, int W, int act, cudaStream_t st) {
  if (kin < 1 || kin > 16 || nout < 1 || nout > 16 || n < 1 || D < 1 || H < 1 || W < 1)
    return cudaErrorInvalidValue;
  const TcGeom G = tc_geom(W);
  cudaError_t e =
      cudaFuncSetAttribute(k_conv_tc<BWD>, cudaFuncAttributeMaxDynamicSharedMemorySize, kTcMaxBytes);
  if (e != cudaSuccess) return e;
  const int ndt = (D + kTcD - 1) / kTcD;
  const dim3 grid((W + G.outc - 1) / G.outc, (H + G.rows - 1) / G.rows, n * ndt);
  k_conv_tc<BWD><<<grid, kTcThreads, G.bytes, st>>>(in, static_cast<const __nv_bfloat16 *>(w), face, z, a,
                                                    kin, nout, D, H, W, ndt, act);
  return cudaGetLastError();
}

}  // namespace

int nn_conv_fwd_tc(const float *in, const void *w_bf16, const int *face, float *z, float *a, int n,
                   int ci, int co, int D, int H, int W, int act, void *stream) {
  return launch_tc<false>(in, w_bf16, face, z, a, n, ci, co, D, H, W, act,
                          static_cast<cudaStream_t>(stream));
}

int nn_conv_bwd_data_tc(const float *dz, const void *w_bf16, const int *face, float *din, int n,
                        int ci, int co, int D, int H, int W, void *stream) {
  return launch_tc<true>(dz, w_bf16, face, nullptr, din, n, co, ci, D, H, W, 0,
                         static_cast<cudaStream_t>(stream));
}

unsigned long long nn_tc_timeouts() {
  unsigned long long v = 0;
  cudaMemcpyFromSymbol(&v, g_tc_timeouts, sizeof(v));
  return v;
}

}  // namespace wf
