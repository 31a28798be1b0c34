// Convolutions of small images with few channels (LeNet's layers), stride 1, exact fp32.  As a matrix product such a layer
// has 6-16 rows: a 64-wide tile multiplies mostly padding and spends its time turning flat indices into addresses
// (the 16 -> 6 channel input gradient at 14x14, batch 256: 283 us for 0.24 GFLOP).  Here a block keeps one image (zero halo
// included) and all filters in shared memory, so an operand costs one shared-memory read and no index arithmetic:
//   forward / input gradient   a thread owns 4 neighbouring outputs of 2 channels: per input channel and filter row two or
//                              three 16-byte reads of the image row feed 8*S multiply-adds.  Bound by FMA issue.
//   filter gradient            a thread owns one (output channel, input channel, filter row) and slides along the image row
//                              with S accumulators: two reads feed S multiply-adds.  Bound by shared-memory reads; images are
//                              dealt to the blocks, whose partial sums are added in block order (bit-reproducible).
#include "common.h"

namespace tf {

struct DirectConv {
  const float* in; const float* w; float* out;
  int N, Ci, Hi, Wi, Co, Ho, Wo, R, S, pad_h, pad_w;
  int flip;                   // input gradient: w is [in][out][R][S], read back to front
  int hp, wp, groups, items;  // halo image, 4-output groups per row, work items of one image
};
constexpr int kPair = 2;

template <int S>
__global__ void __launch_bounds__(256) direct_conv_kernel(const DirectConv p, AmaxOut am) {
  extern __shared__ __align__(16) float direct_smem[];
  float* xs = direct_smem;                                     // [Ci][hp][wp]
  float* ws = direct_smem + p.Ci * p.hp * p.wp;                // [channel pair][Ci][R][S][2]
  grid_dep_sync();
  const int n = blockIdx.x, pairs = (p.Co + kPair - 1) / kPair, rs = p.R * S;
  const float* src = p.in + (long long)n * p.Ci * p.Hi * p.Wi;
  for (int i = threadIdx.x; i < p.Ci * p.hp * p.wp; i += blockDim.x) {
    const int c = i / (p.hp * p.wp), rem = i - c * p.hp * p.wp, y = rem / p.wp - p.pad_h, x = rem % p.wp - p.pad_w;
    xs[i] = (unsigned)y < (unsigned)p.Hi && (unsigned)x < (unsigned)p.Wi ? __ldg(src + (c * p.Hi + y) * p.Wi + x) : 0.f;
  }
  for (int i = threadIdx.x; i < pairs * p.Ci * rs * kPair; i += blockDim.x) {
    const int o2 = i % kPair, t = (i / kPair) % rs, ci = (i / (kPair * rs)) % p.Ci, o = i / (kPair * rs * p.Ci) * kPair + o2;
    float v = 0.f;
    if (o < p.Co) v = __ldg(p.flip ? p.w + ((long long)ci * p.Co + o) * rs + (rs - 1 - t) : p.w + ((long long)o * p.Ci + ci) * rs + t);
    ws[i] = v;
  }
  __syncthreads();
  uint32_t big = 0;
  for (int item = blockIdx.y * blockDim.x + threadIdx.x; item < p.items; item += gridDim.y * blockDim.x) {
    const int g = item % p.groups, row = (item / p.groups) % p.Ho, pair = item / (p.groups * p.Ho);
    float acc[kPair][4];
#pragma unroll
    for (int a = 0; a < kPair; ++a)
#pragma unroll
      for (int q = 0; q < 4; ++q) acc[a][q] = 0.f;
    const float* wp = ws + (long long)pair * p.Ci * rs * kPair;
    for (int ci = 0; ci < p.Ci; ++ci) {
      const float* xr = xs + (ci * p.hp + row) * p.wp + 4 * g;
      for (int r = 0; r < p.R; ++r, xr += p.wp, wp += S * kPair) {
        constexpr int kVec = (S + 3 + 3) / 4;
        float x[4 * kVec];
#pragma unroll
        for (int v = 0; v < kVec; ++v) *reinterpret_cast<float4*>(x + 4 * v) = *reinterpret_cast<const float4*>(xr + 4 * v);
#pragma unroll
        for (int s = 0; s < S; ++s) {
          const float2 f = *reinterpret_cast<const float2*>(wp + s * kPair);
#pragma unroll
          for (int q = 0; q < 4; ++q) { acc[0][q] = fmaf(x[s + q], f.x, acc[0][q]); acc[1][q] = fmaf(x[s + q], f.y, acc[1][q]); }
        }
      }
    }
#pragma unroll
    for (int a = 0; a < kPair; ++a) {
      const int o = pair * kPair + a;
      if (o >= p.Co) continue;
      float* dst = p.out + (((long long)n * p.Co + o) * p.Ho + row) * p.Wo + 4 * g;
#pragma unroll
      for (int q = 0; q < 4; ++q) if (4 * g + q < p.Wo) { dst[q] = acc[a][q]; big = max(big, amax_bits(acc[a][q])); }
    }
  }
  amax_commit(am, big);
}

struct DirectWgrad {
  const float* x; const float* dy; float* part;
  int N, C, H, W, K, P, Q, R, pad_h, pad_w;
  int hp, wp, items, slices, rows_per_slice;
};
constexpr int kWgradThreads = 512, kWgradItems = 4;

template <int S, int IT>
__global__ void __launch_bounds__(kWgradThreads) direct_wgrad_kernel(const DirectWgrad p) {
  extern __shared__ __align__(16) float direct_smem[];
  float* xs = direct_smem;                          // [C][hp][wp]
  float* ds = direct_smem + p.C * p.hp * p.wp;      // [K][P][Q]
  grid_dep_sync();
  const int slice = IT == 1 ? threadIdx.x / p.items : 0, first = IT == 1 ? threadIdx.x - slice * p.items : threadIdx.x;
  const bool live = slice < p.slices;
  float acc[IT][S];
#pragma unroll
  for (int i = 0; i < IT; ++i)
#pragma unroll
    for (int s = 0; s < S; ++s) acc[i][s] = 0.f;
  for (int n = blockIdx.x; n < p.N; n += gridDim.x) {
    __syncthreads();
    const float* xsrc = p.x + (long long)n * p.C * p.H * p.W;
    const float* dsrc = p.dy + (long long)n * p.K * p.P * p.Q;
    for (int i = threadIdx.x; i < p.C * p.hp * p.wp; i += blockDim.x) {
      const int c = i / (p.hp * p.wp), rem = i - c * p.hp * p.wp, y = rem / p.wp - p.pad_h, x = rem % p.wp - p.pad_w;
      xs[i] = (unsigned)y < (unsigned)p.H && (unsigned)x < (unsigned)p.W ? __ldg(xsrc + (c * p.H + y) * p.W + x) : 0.f;
    }
    for (int i = threadIdx.x; i < p.K * p.P * p.Q; i += blockDim.x) ds[i] = __ldg(dsrc + i);
    __syncthreads();
#pragma unroll
    for (int it = 0; it < IT; ++it) {
      const int item = first + it * kWgradThreads;
      if (!live || item >= p.items) continue;
      const int r = item % p.R, c = (item / p.R) % p.C, k = item / (p.R * p.C);
      const int p0 = slice * p.rows_per_slice, p1 = min(p.P, p0 + p.rows_per_slice);
      for (int pp = p0; pp < p1; ++pp) {
        const float* xr = xs + (c * p.hp + pp + r) * p.wp;
        const float* dr = ds + (k * p.P + pp) * p.Q;
        float win[S];
#pragma unroll
        for (int s = 0; s < S - 1; ++s) win[s] = xr[s];
        for (int q = 0; q < p.Q; ++q) {
          win[S - 1] = xr[q + S - 1];
          const float d = dr[q];
#pragma unroll
          for (int s = 0; s < S; ++s) acc[it][s] = fmaf(win[s], d, acc[it][s]);
#pragma unroll
          for (int s = 0; s < S - 1; ++s) win[s] = win[s + 1];
        }
      }
    }
  }
  float* out = p.part + (long long)blockIdx.x * p.items * S;
  if (IT > 1 || p.slices == 1) {
#pragma unroll
    for (int it = 0; it < IT; ++it) {
      const int item = first + it * kWgradThreads;
      if (!live || item >= p.items) continue;
#pragma unroll
      for (int s = 0; s < S; ++s) out[item * S + s] = acc[it][s];
    }
    return;
  }
  __syncthreads();
  if (live) {
#pragma unroll
    for (int s = 0; s < S; ++s) direct_smem[(slice * p.items + first) * S + s] = acc[0][s];
  }
  __syncthreads();
  for (int i = threadIdx.x; i < p.items * S; i += blockDim.x) {
    float t = 0.f;
    for (int z = 0; z < p.slices; ++z) t += direct_smem[z * p.items * S + i];
    out[i] = t;
  }
}
// out[c] = sum over the blocks' partial filters, in block order within each of 8 lanes
__global__ void __launch_bounds__(256) direct_wgrad_sum_kernel(const float* __restrict__ part, float* __restrict__ out, int rows, int cols) {
  __shared__ float sm[8][33];
  grid_dep_sync();
  const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5, c = blockIdx.x * 32 + tx;
  float acc = 0.f;
  if (c < cols) {
#pragma unroll 4
    for (int r = ty; r < rows; r += 8) acc += part[(long long)r * cols + c];
  }
  sm[ty][tx] = acc;
  __syncthreads();
  if (ty == 0 && c < cols) {
    float t = 0.f;
#pragma unroll
    for (int j = 0; j < 8; ++j) t += sm[j][tx];
    out[c] = t;
  }
}

constexpr size_t kDirectSmem = 96 * 1024;
// The layers taken: stride 1, windows 3, 5 or 7 wide, an image that fits in shared memory together with the filters, and few
// enough channels that the tensor path would multiply padding (it takes 16 channels and more, in multiples of 4; its first
// layers of three channels have large images and many filters and stay there).
static bool direct_shape(const ConvPlan* p) {
  return p->dataformat == 0 && p->stride_h == 1 && p->stride_w == 1 && (p->S == 3 || p->S == 5 || p->S == 7) && p->R <= 7 && p->pad_h <= p->R - 1 && p->pad_w <= p->S - 1 &&
         p->K <= 32 && p->C <= 32 && (p->C < 16 || p->K < 16) && (long long)p->K * p->C * p->R * p->S <= 8192 && p->P == p->H + 2 * p->pad_h - p->R + 1 && p->Q == p->W + 2 * p->pad_w - p->S + 1;
}
static int launch_direct(DirectConv d, cudaStream_t s, double flops, const char* what) {
  d.groups = (d.Wo + 3) / 4;
  d.hp = d.Ho + d.R - 1;
  d.wp = (4 * d.groups + d.S + 2) / 4 * 4;           // every 16-byte read of the last group stays inside the row
  d.items = (d.Co + kPair - 1) / kPair * d.Ho * d.groups;
  const size_t smem = sizeof(float) * ((size_t)d.Ci * d.hp * d.wp + (size_t)(d.Co + 1) / 2 * 2 * d.Ci * d.R * d.S);
  if (smem > kDirectSmem) return 0;
  // one block per image unless that leaves SMs idle
  int gy = (d.items + 255) / 256;
  while (gy > 1 && (long long)d.N * (gy - 1) >= 4 * device_sm_count()) --gy;
  if (gy > 65535) gy = 65535;
  note_compute_stream(s);
  KernelTimer kt("direct_conv", s, flops, 0, 1);
  auto kernel = d.S == 3 ? direct_conv_kernel<3> : d.S == 5 ? direct_conv_kernel<5> : direct_conv_kernel<7>;
  TF_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kDirectSmem));
  TF_CUDA(launch_dep(kernel, dim3(d.N, gy), dim3(256), smem, s, d, amax_track_begin(d.out)));
  TF_AFTER(s, what);
  return 1;
}
// Each returns 1 when it took the call, 0 when the shape is not one of its own, -1 on error.
int direct_conv_fwd(const ConvPlan* p, const float* x, const float* w, float* y, cudaStream_t s) {
  if (!direct_shape(p)) return 0;
  DirectConv d{x, w, y, p->N, p->C, p->H, p->W, p->K, p->P, p->Q, p->R, p->S, p->pad_h, p->pad_w, 0, 0, 0, 0, 0};
  return launch_direct(d, s, 2.0 * p->N * p->K * p->P * p->Q * p->C * p->R * p->S, "DLGpuConvolution2DForward");
}
int direct_conv_dgrad(const ConvPlan* p, const float* dy, const float* w, float* dx, cudaStream_t s) {
  if (!direct_shape(p)) return 0;
  DirectConv d{dy, w, dx, p->N, p->K, p->P, p->Q, p->C, p->H, p->W, p->R, p->S, p->R - 1 - p->pad_h, p->S - 1 - p->pad_w, 1, 0, 0, 0, 0};
  return launch_direct(d, s, 2.0 * p->N * p->K * p->P * p->Q * p->C * p->R * p->S, "DLGpuConvolutionBackwardData");
}
template <int S> static int launch_wgrad(const DirectWgrad& d, int grid, size_t smem, cudaStream_t s) {
  const int per = (d.items + kWgradThreads - 1) / kWgradThreads;
  auto kernel = per <= 1 ? direct_wgrad_kernel<S, 1> : per <= 2 ? direct_wgrad_kernel<S, 2> : direct_wgrad_kernel<S, kWgradItems>;
  TF_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kDirectSmem));
  TF_CUDA(launch_dep(kernel, dim3(grid), dim3(kWgradThreads), smem, s, d));
  return 0;
}
int direct_conv_wgrad(const ConvPlan* p, const float* x, const float* dy, float* dw, cudaStream_t s) {
  if (!direct_shape(p) || p->K * p->C * p->R > kWgradThreads * kWgradItems) return 0;
  DirectWgrad d{x, dy, nullptr, p->N, p->C, p->H, p->W, p->K, p->P, p->Q, p->R, p->pad_h, p->pad_w, p->P + p->R - 1, 0, p->K * p->C * p->R, 1, p->P};
  d.wp = (p->Q + p->S - 1) | 1;                 // odd pitch: the filter rows of a warp fall in different banks
  if (d.items <= kWgradThreads) {               // threads to spare: cut the image rows
    d.slices = kWgradThreads / d.items;
    if (d.slices > p->P) d.slices = p->P;
    d.rows_per_slice = (p->P + d.slices - 1) / d.slices;
  }
  size_t floats = (size_t)p->C * d.hp * d.wp + (size_t)p->K * p->P * p->Q;
  if (d.slices > 1 && floats < (size_t)d.slices * d.items * p->S) floats = (size_t)d.slices * d.items * p->S;
  if (floats * sizeof(float) > kDirectSmem) return 0;
  const int cols = d.items * p->S, grid = p->N < 2 * device_sm_count() ? p->N : 2 * device_sm_count();
  StreamLease lease(s);
  d.part = (float*)lease.scratch(kScratchContract, sizeof(float) * (size_t)grid * cols);
  if (!d.part) return 0;
  note_compute_stream(s);
  KernelTimer kt("direct_conv", s, 2.0 * p->N * p->K * p->P * p->Q * p->C * p->R * p->S, 0, 1);
  if ((p->S == 3 ? launch_wgrad<3>(d, grid, floats * sizeof(float), s) : p->S == 5 ? launch_wgrad<5>(d, grid, floats * sizeof(float), s) : launch_wgrad<7>(d, grid, floats * sizeof(float), s)) != 0) return -1;
  TF_AFTER(s, "DLGpuConvolutionBackwardFilter");
  TF_CUDA(launch_dep(direct_wgrad_sum_kernel, dim3((cols + 31) / 32), dim3(256), 0, s, (const float*)d.part, dw, grid, cols));
  TF_AFTER(s, "DLGpuConvolutionBackwardFilter");
  return 1;
}

}  // namespace tf
