// Element-wise kernels of the inference forward (CrossLayerTranscoder.forward and the per-layer
// forward_layer calls of the reference, crosslayer_transcoder/model/clt.py:134-145, 216-231, 304-317,
// 403-425): layout changes between the token-major tensors of the module surface and the layer-major
// operands of the contraction kernels, with the bias / statistics applied on the way.
#include "../../include/clt_b200.h"
#include "common.cuh"
#include "kernels.h"

namespace clt {
namespace {

// Rows of V consecutive elements in registers; V = 8 needs rows that start on 32-byte boundaries.
template <class T, int V>
__device__ __forceinline__ void load_row(const T* p, float (&o)[V]) {
  if constexpr (V == 1) {
    if constexpr (sizeof(T) == 2)
      o[0] = __bfloat162float(*p);
    else
      o[0] = *p;
  } else if constexpr (sizeof(T) == 2) {
    const uint4 t = __ldcs(reinterpret_cast<const uint4*>(p));
    const uint32_t w[4] = {t.x, t.y, t.z, t.w};
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      o[2 * j] = __uint_as_float(w[j] << 16);
      o[2 * j + 1] = __uint_as_float(w[j] & 0xffff0000u);
    }
  } else {
    const float4 a = __ldcs(reinterpret_cast<const float4*>(p)), b = __ldcs(reinterpret_cast<const float4*>(p) + 1);
    o[0] = a.x, o[1] = a.y, o[2] = a.z, o[3] = a.w, o[4] = b.x, o[5] = b.y, o[6] = b.z, o[7] = b.w;
  }
}
template <class T, int V>
__device__ __forceinline__ void store_row(T* p, const float (&v)[V]) {
  if constexpr (V == 1) {
    if constexpr (sizeof(T) == 2)
      *p = __float2bfloat16_rn(v[0]);
    else
      *p = v[0];
  } else if constexpr (sizeof(T) == 2) {
    *reinterpret_cast<uint4*>(p) = make_uint4(pack_bf16x2(v[0], v[1]), pack_bf16x2(v[2], v[3]),
                                              pack_bf16x2(v[4], v[5]), pack_bf16x2(v[6], v[7]));
  } else {
    st_f32x8(p, make_float4(v[0], v[1], v[2], v[3]), make_float4(v[4], v[5], v[6], v[7]));
  }
}
template <class T>
__device__ __forceinline__ float rounded(float x) {
  return sizeof(T) == 2 ? bf16_round(x) : x;
}

// The three layout kernels below are bound by HBM.  A CTA covers 256 V columns of one layer (blockIdx.x, blockIdx.z)
// and walks batch rows (blockIdx.y strided), so an element costs no division and the per-column parameters stay in
// registers; V = 8 makes every load 16 and every fp32 store 32 bytes wide, V = 1 takes the rows that do not start on
// such boundaries.  export at [12, 1000, 10000] bf16:
// 472 -> 128 us (5.6 TB/s; 162 us with two 16-byte stores), one element per thread and step with two 64-bit divisions
// before; act_export at [12, 333, 24576] 195 us (6.0 TB/s) for what an activation sweep and two exports took 900 us.

// out[b, l, f] = src[l, b, f] (+ bias[l, f])     layer-major T -> token-major fp32
template <class T, int V>
__global__ void __launch_bounds__(256)
export_blf_kernel(const T* __restrict__ src, const float* __restrict__ bias, float* __restrict__ out, int B, int L,
                  long long F) {
  const long long f = (blockIdx.x * 256ll + threadIdx.x) * V;
  const int l = blockIdx.z;
  if (f >= F) return;
  float bb[V];
#pragma unroll
  for (int q = 0; q < V; ++q) bb[q] = 0.f;
  if (bias != nullptr) {
#pragma unroll
    for (int q = 0; q < V; ++q) bb[q] = __ldg(bias + l * F + f + q);
  }
#pragma unroll 2
  for (int b = blockIdx.y; b < B; b += gridDim.y) {
    float v[V];
    load_row<T, V>(src + ((long long)l * B + b) * F + f, v);
    if (bias != nullptr) {
#pragma unroll
      for (int q = 0; q < V; ++q) v[q] += bb[q];
    }
    store_row<float, V>(out + ((long long)b * L + l) * F + f, v);
  }
}

// pre[b, l, f] = z[l, b, f] + bias[l, f];  feat[l, b, f] = T(pre [pre > theta, pre > 0]);  features[b, l, f] = feat:
// the validation forward's (Jump)ReLU and both of its token-major outputs from one sweep of z
template <class T, int V>
__global__ void __launch_bounds__(256)
act_export_kernel(const T* __restrict__ z, const float* __restrict__ bias, const float* __restrict__ theta,
                  float* __restrict__ pre, T* __restrict__ feat, float* __restrict__ features, int B, int L,
                  long long F) {
  const long long f = (blockIdx.x * 256ll + threadIdx.x) * V;
  const int l = blockIdx.z;
  if (f >= F) return;
  float bb[V], tt[V];
#pragma unroll
  for (int q = 0; q < V; ++q) {
    bb[q] = __ldg(bias + l * F + f + q);
    tt[q] = theta != nullptr ? __ldg(theta + l * F + f + q) : 0.f;
  }
#pragma unroll 2
  for (int b = blockIdx.y; b < B; b += gridDim.y) {
    const long long lm = ((long long)l * B + b) * F + f, tm = ((long long)b * L + l) * F + f;
    float v[V], a[V];
    load_row<T, V>(z + lm, v);
#pragma unroll
    for (int q = 0; q < V; ++q) {
      v[q] += bb[q];
      a[q] = rounded<T>(v[q] > tt[q] && v[q] > 0.f ? v[q] : 0.f);
    }
    store_row<float, V>(pre + tm, v);
    store_row<T, V>(feat + lm, a);
    store_row<float, V>(features + tm, a);
  }
}

// dst[l, b, f] = T(src[b * ld + l * F + f])       fp32 rows of any distance -> layer-major T
template <class T, int V>
__global__ void __launch_bounds__(256)
import_rows_kernel(const float* __restrict__ src, long long ld, T* __restrict__ dst, int B, long long F) {
  const long long f = (blockIdx.x * 256ll + threadIdx.x) * V;
  const int l = blockIdx.z;
  if (f >= F) return;
#pragma unroll 2
  for (int b = blockIdx.y; b < B; b += gridDim.y) {
    float v[V];
    load_row<float, V>(src + (long long)b * ld + l * F + f, v);
    store_row<T, V>(dst + ((long long)l * B + b) * F + f, v);
  }
}

// grid of these kernels for CTAs `wide` columns wide: about 16 CTAs per SM, fewer rows per CTA rather than fewer CTAs
inline dim3 row_grid(int B, int L, long long F, long long wide) {
  const long long gx = (F + wide - 1) / wide;
  long long gy = (148ll * 16 + gx * L - 1) / (gx * L);
  if (gy > B) gy = B;
  return dim3((unsigned)gx, (unsigned)(gy < 65535 ? gy : 65535), (unsigned)L);
}
template <class T>
int launch_import(const float* src, long long ld, void* dst, int B, int L, long long F, cudaStream_t s) {
  if (F % 8 == 0 && ld % 8 == 0 && aligned32(src) && aligned32(dst))
    import_rows_kernel<T, 8><<<row_grid(B, L, F, 256 * 8), 256, 0, s>>>(src, ld, (T*)dst, B, F);
  else
    import_rows_kernel<T, 1><<<row_grid(B, L, F, 256), 256, 0, s>>>(src, ld, (T*)dst, B, F);
  CLT_CHECK_CUDA(cudaGetLastError());
  return 0;
}
template <class T>
int launch_export(const void* src, const float* bias, float* out, int B, int L, long long F, cudaStream_t s) {
  if (F % 8 == 0 && aligned32(src) && aligned32(out))
    export_blf_kernel<T, 8><<<row_grid(B, L, F, 256 * 8), 256, 0, s>>>((const T*)src, bias, out, B, L, F);
  else
    export_blf_kernel<T, 1><<<row_grid(B, L, F, 256), 256, 0, s>>>((const T*)src, bias, out, B, L, F);
  CLT_CHECK_CUDA(cudaGetLastError());
  return 0;
}
template <class T>
int launch_act_export(const void* z, const float* bias, const float* theta, float* pre, void* feat, float* features,
                      int B, int L, long long F, cudaStream_t s) {
  if (F % 8 == 0 && aligned32(z) && aligned32(pre) && aligned32(feat) && aligned32(features))
    act_export_kernel<T, 8>
        <<<row_grid(B, L, F, 256 * 8), 256, 0, s>>>((const T*)z, bias, theta, pre, (T*)feat, features, B, L, F);
  else
    act_export_kernel<T, 1>
        <<<row_grid(B, L, F, 256), 256, 0, s>>>((const T*)z, bias, theta, pre, (T*)feat, features, B, L, F);
  CLT_CHECK_CUDA(cudaGetLastError());
  return 0;
}

// out[b, l, d] = recon[b, l, d] * sd[l, d] + mu[l, d].  A CTA's x covers V columns a thread of the L D of a row, its y (where
// rows are narrower than 256 threads) and blockIdx.y walk rows, so that the statistics stay in registers and an element
// costs no 64-bit division (inputs not in L2: 1000 x 12 x 768 33 -> 18 us, 4.1 TB/s; 1500 x 12 x 2304 112 -> 64 us, 5.2
// TB/s).  V = 4: 16-byte accesses.
template <int V>
__global__ void __launch_bounds__(256)
destandardize_kernel(const float* __restrict__ recon, const float* __restrict__ mu, const float* __restrict__ sd,
                     float* __restrict__ out, int B, long long LD) {
  const long long c = (blockIdx.x * (long long)blockDim.x + threadIdx.x) * V;
  if (c >= LD) return;
  float m[V], d[V];
#pragma unroll
  for (int q = 0; q < V; ++q) m[q] = __ldg(mu + c + q), d[q] = __ldg(sd + c + q);
#pragma unroll 4
  for (long long b = blockIdx.y * blockDim.y + threadIdx.y; b < B; b += gridDim.y * blockDim.y) {
    const long long i = b * LD + c;
    if constexpr (V == 4) {
      const float4 r = *reinterpret_cast<const float4*>(recon + i);
      *reinterpret_cast<float4*>(out + i) =
          make_float4(fmaf(r.x, d[0], m[0]), fmaf(r.y, d[1], m[1]), fmaf(r.z, d[2], m[2]), fmaf(r.w, d[3], m[3]));
    } else {
      out[i] = fmaf(recon[i], d[0], m[0]);
    }
  }
}
template <int V>
int launch_destandardize(const float* recon, const float* mu, const float* sd, float* out, int B, long long LD,
                         cudaStream_t s) {
  const long long cols = (LD + V - 1) / V;
  int x = 256;
  while (x > 1 && x / 2 >= cols) x /= 2;
  const dim3 block(x, 256 / x);
  const dim3 grid = row_grid((B + (int)block.y - 1) / (int)block.y, 1, LD, x * V);
  destandardize_kernel<V><<<grid, block, 0, s>>>(recon, mu, sd, out, B, LD);
  CLT_CHECK_CUDA(cudaGetLastError());
  return 0;
}

// dense[token, l, idx] = val for every valid entry of the per-layer lists idx / val [L, npl]; the token of
// entry e is etok[e], or e / k for the fixed-slot lists of the per-row selection (npl = B k)
__global__ void scatter_features_kernel(const int* __restrict__ idx, const float* __restrict__ val,
                                        const int* __restrict__ etok, float* __restrict__ dense, int B, int L, int F,
                                        int k, long long npl, int* status) {
  const long long total = (long long)L * npl;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < total;
       i += (long long)gridDim.x * blockDim.x) {
    const float v = val[i];
    if (v == 0.f) continue;
    const int f = idx[i];
    const int l = (int)(i / npl);
    const long long b = etok != nullptr ? (long long)etok[i] : (i - (long long)l * npl) / k;
    if (f < 0 || f >= F || b < 0 || b >= B) {
      report_status(status, kBadIndex);
      continue;
    }
    dense[(b * L + l) * (long long)F + f] = v;
  }
}

inline unsigned grid_for(long long total) {
  const long long want = (total + 255) / 256;
  return (unsigned)(want < 148 * 16 ? (want > 0 ? want : 1) : 148 * 16);
}

}  // namespace
}  // namespace clt

using namespace clt;

extern "C" {

int clt_prep_acts(const void* acts, int in_dtype, const float* mu, const float* sd, void* xn, int bf16, int B, int L,
                  int D, clt_stream_t stream) {
  CLT_CHECK_ARG(acts && xn && B > 0 && L > 0 && D > 0, "prep_acts: bad arguments");
  CLT_CHECK_ARG((mu == nullptr) == (sd == nullptr), "prep_acts: mean and std go together");
  return prep_input(acts, in_dtype, mu, sd, xn, bf16, B, L, D, 1, (cudaStream_t)stream);
}

int clt_export_blf(const void* src, const float* bias, float* out, int B, int L, int64_t F, int bf16,
                   clt_stream_t stream) {
  CLT_CHECK_ARG(src && out && B > 0 && L > 0 && L <= 65535 && F > 0, "export_blf: bad arguments");
  return bf16 ? launch_export<__nv_bfloat16>(src, bias, out, B, L, F, (cudaStream_t)stream)
              : launch_export<float>(src, bias, out, B, L, F, (cudaStream_t)stream);
}

int clt_act_export(const void* z, const float* bias, const float* theta, float* pre, void* feat, float* features, int B,
                   int L, int64_t F, int bf16, clt_stream_t stream) {
  CLT_CHECK_ARG(z && bias && pre && feat && features && B > 0 && L > 0 && L <= 65535 && F > 0,
                "act_export: bad arguments");
  return bf16 ? launch_act_export<__nv_bfloat16>(z, bias, theta, pre, feat, features, B, L, F, (cudaStream_t)stream)
              : launch_act_export<float>(z, bias, theta, pre, feat, features, B, L, F, (cudaStream_t)stream);
}

int clt_import_blf(const float* src, void* dst, int B, int L, int64_t F, int bf16, clt_stream_t stream) {
  CLT_CHECK_ARG(src && dst && B > 0 && L > 0 && L <= 65535 && F > 0, "import_blf: bad arguments");
  const long long ld = (long long)L * F;
  return bf16 ? launch_import<__nv_bfloat16>(src, ld, dst, B, L, F, (cudaStream_t)stream)
              : launch_import<float>(src, ld, dst, B, L, F, (cudaStream_t)stream);
}

int clt_import_rows(const float* src, int64_t ld, void* dst, int rows, int64_t K, int bf16, clt_stream_t stream) {
  CLT_CHECK_ARG(src && dst && rows > 0 && K > 0 && ld >= 0, "import_rows: bad arguments");
  return bf16 ? launch_import<__nv_bfloat16>(src, ld, dst, rows, 1, K, (cudaStream_t)stream)
              : launch_import<float>(src, ld, dst, rows, 1, K, (cudaStream_t)stream);
}

int clt_destandardize(const float* recon, const float* mu, const float* sd, float* out, int B, int L, int D,
                      clt_stream_t stream) {
  CLT_CHECK_ARG(recon && mu && sd && out && B > 0 && L > 0 && D > 0, "destandardize: bad arguments");
  const long long LD = (long long)L * D;
  const int V = LD % 4 == 0 && ((uintptr_t)recon | (uintptr_t)out) % 16 == 0 ? 4 : 1;
  return V == 4 ? launch_destandardize<4>(recon, mu, sd, out, B, LD, (cudaStream_t)stream)
                : launch_destandardize<1>(recon, mu, sd, out, B, LD, (cudaStream_t)stream);
}

int clt_scatter_features(const int* idx, const float* val, const int* etok, float* dense, int B, int L, int F, int k,
                         int64_t npl, int* status, clt_stream_t stream) {
  CLT_CHECK_ARG(idx && val && dense && B > 0 && L > 0 && F > 0 && k > 0 && npl > 0, "scatter_features: bad arguments");
  CLT_CHECK_ARG(etok != nullptr || npl == (int64_t)B * k, "scatter_features: fixed slots need npl = B*k");
  cudaStream_t s = (cudaStream_t)stream;
  CLT_CHECK_CUDA(cudaMemsetAsync(dense, 0, sizeof(float) * (size_t)B * L * F, s));
  scatter_features_kernel<<<grid_for((long long)L * npl), 256, 0, s>>>(idx, val, etok, dense, B, L, F, k, npl, status);
  CLT_CHECK_CUDA(cudaGetLastError());
  return 0;
}

}  // extern "C"
