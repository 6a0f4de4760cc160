// fp32 contraction on the CUDA cores, for the fp32 configuration whose parity
// bar (1e-4 relative) a single-pass tensor-core format cannot meet.
//
// Bound by the fp32 pipes: 256 threads compute a tile of 16*TM x 16*TN, a thread TM x TN of it as
// packed pairs along n (fma.rn.f32x2: half the issue slots of scalar FMAs, same rounding), so that at
// TM = TN = 8 a k-step is 32 packed FMAs beside 4 shared-memory loads.  Operand tiles of 16 k-steps are
// double-buffered: the global loads of the next tile are in flight, in registers, while the current one
// is multiplied, and every load is 16 bytes along the operand's contiguous axis where its strides allow.
// Each output is one fma chain in ascending k, whatever the tile.
// 12-layer, 1024-feature, 512-token JumpReLU step (its five contractions): 12.6 -> 5.3 ms, 4.8 with the decoder in
// parts and the feature gradient in half tiles; the kernel before gave a thread one row x 64 columns, read K-contiguous
// operands 4 bytes a row, and loaded and multiplied in turn.  At 8 x 8 the plain epilogue needs 126 registers; those of
// the (Jump)ReLU spill around it (104 bytes forward, 812 backward, where half tiles spill none).
//
// The finished tile goes through shared memory, 64 columns at a time, into the shape that the
// tcgen05 kernel reads out of tensor memory (a warp holds 32 rows, a lane 32 columns of its row), so
// both kernels share their epilogue functors.
#pragma once

#include "epilogues.cuh"
#include "gemm.cuh"

namespace clt {

struct SimtOperands {
  const float* A;
  const float* B;
  // element strides: A(za, m, k) = A[za*sAz + m*sAm + k*sAk], B(zb, k, n) = B[zb*sBz + k*sBk + n*sBn]
  long long sAz, sAm, sAk;
  long long sBz, sBk, sBn;
  int vecA, vecB;  // every 4 elements along the contiguous axis are one aligned 16-byte load
};

constexpr int kSimtThreads = 256, kSimtBK = 16;
constexpr int kSimtSubLd = 36;                       // row stride of a 32 x 32 sub-tile on its way to the epilogue
constexpr int kSimtSubFloats = 32 * kSimtSubLd;
static_assert(kSimtSubFloats * 4 >= epi::kStageBytes, "a sub-tile's memory doubles as its warp's store staging");

// One operand tile of MN x 16 (k), as this thread's share in registers: 16-byte pieces along the
// contiguous axis, or single elements when rows are not 16-byte aligned.  Elements outside read as 0.
template <int MN>
struct SimtTile {
  static constexpr int kPer = MN * kSimtBK / kSimtThreads;  // values per thread (8 or 4)
  static constexpr int kLd = MN + 4;
  float r[kPer];

  __device__ __forceinline__ void load(const float* __restrict__ p, long long s_mn, long long s_k, bool vec, int mn0,
                                       int n_mn, int k0, int n_k) {
    const int tid = threadIdx.x;
    const bool kc = s_k == 1;
    if (vec) {
#pragma unroll
      for (int i = 0; i < kPer / 4; ++i) {
        const int e = tid + kSimtThreads * i;
        const int mn = kc ? e >> 2 : (e % (MN / 4)) * 4;
        const int k = kc ? (e & 3) * 4 : e / (MN / 4);
        float4 t = make_float4(0.f, 0.f, 0.f, 0.f);
        if (mn0 + mn < n_mn && k0 + k < n_k)
          t = __ldg(reinterpret_cast<const float4*>(p + (long long)(mn0 + mn) * s_mn + (long long)(k0 + k) * s_k));
        r[4 * i] = t.x, r[4 * i + 1] = t.y, r[4 * i + 2] = t.z, r[4 * i + 3] = t.w;
      }
    } else {
#pragma unroll
      for (int i = 0; i < kPer; ++i) {
        const int e = tid + kSimtThreads * i;
        const int mn = kc ? e / kSimtBK : e % MN;
        const int k = kc ? e % kSimtBK : e / MN;
        r[i] = (mn0 + mn < n_mn && k0 + k < n_k)
                   ? __ldg(p + (long long)(mn0 + mn) * s_mn + (long long)(k0 + k) * s_k)
                   : 0.f;
      }
    }
  }

  // sm[k][mn], row stride kLd
  __device__ __forceinline__ void store(float* sm, bool kc, bool vec) const {
    const int tid = threadIdx.x;
    if (vec) {
#pragma unroll
      for (int i = 0; i < kPer / 4; ++i) {
        const int e = tid + kSimtThreads * i;
        if (kc) {
          float* d = sm + (e & 3) * 4 * kLd + (e >> 2);
#pragma unroll
          for (int j = 0; j < 4; ++j) d[j * kLd] = r[4 * i + j];
        } else {
          *reinterpret_cast<float4*>(sm + (e / (MN / 4)) * kLd + (e % (MN / 4)) * 4) =
              make_float4(r[4 * i], r[4 * i + 1], r[4 * i + 2], r[4 * i + 3]);
        }
      }
    } else {
#pragma unroll
      for (int i = 0; i < kPer; ++i) {
        const int e = tid + kSimtThreads * i;
        const int mn = kc ? e / kSimtBK : e % MN;
        const int k = kc ? e % kSimtBK : e / MN;
        sm[k * kLd + mn] = r[i];
      }
    }
  }
};

typedef unsigned long long f32x2_t;
__device__ __forceinline__ f32x2_t pack_f32x2(float lo, float hi) {
  f32x2_t r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
  return r;
}
__device__ __forceinline__ void unpack_f32x2(f32x2_t v, float& lo, float& hi) {
  asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v));
}
__device__ __forceinline__ void fma_f32x2(f32x2_t& d, f32x2_t a, f32x2_t b) {
  asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(d) : "l"(a), "l"(b));
}

template <int TM, int TN>
struct SimtSmem {
  static constexpr int kOperands = 2 * kSimtBK * (SimtTile<16 * TM>::kLd + SimtTile<16 * TN>::kLd);
  static constexpr int kSubtiles = (TM / 2) * 2 * kSimtSubFloats;
  static constexpr int kFloats = kOperands > kSubtiles ? kOperands : kSubtiles;
};

template <class Epi, int TM, int TN>
__global__ void __launch_bounds__(kSimtThreads, 2) gemm_simt_kernel(GemmGeom g, SimtOperands op,
                                                                    typename Epi::Params ep) {
  constexpr int BM = 16 * TM, BN = 16 * TN;
  using TileA = SimtTile<BM>;
  using TileB = SimtTile<BN>;
  __shared__ __align__(16) float smem[SimtSmem<TM, TN>::kFloats];
  constexpr int kCols = Epi::kColArrays > 0 ? Epi::kColArrays : 1;
  __shared__ __align__(16) float colp[kCols][BN];
  auto As = [&](int buf) { return smem + buf * kSimtBK * TileA::kLd; };
  auto Bs = [&](int buf) { return smem + 2 * kSimtBK * TileA::kLd + buf * kSimtBK * TileB::kLd; };

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int kt_per_seg = (g.Kseg + kSimtBK - 1) / kSimtBK;
  int zi, kt_lo, kt_hi, z;  // operand slab, its k-tiles, output slab
  work_item(g, blockIdx.z, kt_per_seg, zi, kt_lo, kt_hi, z);
  const int m0 = blockIdx.y * BM;
  const int n0 = blockIdx.x * BN;
  // a warp covers 4 x 8 threads: its fragments are 64 and 128 contiguous bytes of a k-row
  const int ty = (warp >> 1) * 4 + (lane >> 3), tx = (warp & 1) * 8 + (lane & 7);

  f32x2_t acc[TM][TN / 2];
#pragma unroll
  for (int i = 0; i < TM; ++i)
#pragma unroll
    for (int j = 0; j < TN / 2; ++j) acc[i][j] = 0ull;

  const bool kcA = op.sAk == 1, kcB = op.sBk == 1;
  const int n_kt = kt_hi - kt_lo;
  TileA ta;
  TileB tb;
  int seg = kt_lo / kt_per_seg, kt = kt_lo % kt_per_seg;  // the k-tile to be loaded next
  const float *Ap = nullptr, *Bp = nullptr;
  auto load_next = [&]() {
    if (kt == 0 || Ap == nullptr) {
      int za, zb;
      seg_index(g, zi, seg, za, zb);
      Ap = op.A + (long long)za * op.sAz;
      Bp = op.B + (long long)zb * op.sBz;
    }
    ta.load(Ap, op.sAm, op.sAk, op.vecA != 0, m0, g.M, kt * kSimtBK, g.Kseg);
    tb.load(Bp, op.sBn, op.sBk, op.vecB != 0, n0, g.N, kt * kSimtBK, g.Kseg);
    if (++kt == kt_per_seg) kt = 0, ++seg;
  };
  if (n_kt > 0) {
    load_next();
    ta.store(As(0), kcA, op.vecA != 0);
    tb.store(Bs(0), kcB, op.vecB != 0);
  }
  __syncthreads();
  for (int it = 0; it < n_kt; ++it) {
    const bool more = it + 1 < n_kt;
    if (more) load_next();
    const float* a_s = As(it & 1) + ty * 4;
    const float* b_s = Bs(it & 1) + tx * 4;
#pragma unroll
    for (int kk = 0; kk < kSimtBK; ++kk) {
      f32x2_t b[TN / 2];
#pragma unroll
      for (int j = 0; j < TN / 4; ++j) {
        const ulonglong2 t = *reinterpret_cast<const ulonglong2*>(b_s + kk * TileB::kLd + 64 * j);
        b[2 * j] = t.x, b[2 * j + 1] = t.y;
      }
#pragma unroll
      for (int i4 = 0; i4 < TM / 4; ++i4) {
        const float4 a4 = *reinterpret_cast<const float4*>(a_s + kk * TileA::kLd + 64 * i4);
        const float av[4] = {a4.x, a4.y, a4.z, a4.w};
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          const f32x2_t a = pack_f32x2(av[q], av[q]);
#pragma unroll
          for (int j = 0; j < TN / 2; ++j) fma_f32x2(acc[4 * i4 + q][j], a, b[j]);
        }
      }
    }
    // the other buffer was last read before the previous barrier
    if (more) {
      ta.store(As((it + 1) & 1), kcA, op.vecA != 0);
      tb.store(Bs((it + 1) & 1), kcB, op.vecB != 0);
    }
    __syncthreads();
  }

  // per-column parameters of this tile, staged once and read as broadcasts
  if (Epi::kColArrays > 0) {
    for (int e = tid; e < Epi::kColArrays * BN; e += kSimtThreads) {
      const int arr = e / BN, j = e % BN;
      colp[arr][j] = (n0 + j < g.N) ? Epi::col_value(ep, arr, z, n0 + j, g.N) : 0.f;
    }
  }
  typename Epi::State st;
  Epi::init(st);
  constexpr int kRowGroups = BM / 32;
#pragma unroll
  for (int h = 0; h < TN / 4; ++h) {  // 64 columns at a time: kRowGroups x 2 sub-tiles, one warp each
#pragma unroll
    for (int i = 0; i < TM; ++i) {
      const int r = (i / 4) * 64 + ty * 4 + (i % 4), c = tx * 4;
      float4 t;
      unpack_f32x2(acc[i][2 * h], t.x, t.y);
      unpack_f32x2(acc[i][2 * h + 1], t.z, t.w);
      *reinterpret_cast<float4*>(smem + ((c >> 5) * kRowGroups + (r >> 5)) * kSimtSubFloats + (r & 31) * kSimtSubLd +
                                 (c & 31)) = t;
    }
    __syncthreads();
    const int chunk = warp / kRowGroups;
    const int nc = n0 + 64 * h + 32 * chunk;
    if (chunk < 2 && nc < g.N) {  // uniform over the warp
      float* sub = smem + warp * kSimtSubFloats;
      float v[32];
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        const float4 t = *reinterpret_cast<const float4*>(sub + lane * kSimtSubLd + 4 * i);
        v[4 * i] = t.x, v[4 * i + 1] = t.y, v[4 * i + 2] = t.z, v[4 * i + 3] = t.w;
      }
      __syncwarp();
      const int row = m0 + 32 * (warp % kRowGroups) + lane;
      Epi::template apply<BN>(ep, st, z, row, row < g.M, nc, g.M, g.N, v, &colp[0][64 * h + 32 * chunk],
                              reinterpret_cast<unsigned char*>(sub));
    }
    __syncthreads();
  }
  Epi::finish(ep, st);
}

template <class Epi, int TM, int TN>
int launch_gemm_simt_tile(const GemmGeom& g, const SimtOperands& op, const typename Epi::Params& ep,
                          cudaStream_t stream) {
  dim3 grid((g.N + 16 * TN - 1) / (16 * TN), (g.M + 16 * TM - 1) / (16 * TM), g.nz);
  CLT_CHECK_ARG(grid.y <= 65535 && grid.z <= 65535, "gemm_simt: grid too large (M=%d nz=%d)", g.M, g.nz);
  gemm_simt_kernel<Epi, TM, TN><<<grid, kSimtThreads, 0, stream>>>(g, op, ep);
  CLT_CHECK_CUDA(cudaGetLastError());
  return 0;
}

template <class Epi>
int launch_gemm_simt(const GemmGeom& g, SimtOperands op, const typename Epi::Params& ep, int num_sms,
                     cudaStream_t stream) {
  if (g.M <= 0 || g.N <= 0 || g.nz <= 0) return 0;
  auto aligned = [](const float* p, long long s_mn, long long s_k, long long s_z) {
    const long long row = s_k == 1 ? s_mn : s_k;  // distance between rows of the contiguous axis
    return ((uintptr_t)p % 16 == 0) && row % 4 == 0 && s_z % 4 == 0;
  };
  // 16-byte loads also need the contiguous axis to end on one
  op.vecA = aligned(op.A, op.sAm, op.sAk, op.sAz) && (op.sAk == 1 ? g.Kseg : g.M) % 4 == 0;
  op.vecB = aligned(op.B, op.sBn, op.sBk, op.sBz) && (op.sBk == 1 ? g.Kseg : g.N) % 4 == 0;
  // Fewer large tiles than SMs leave part of the chip idle: quarter tiles then (each output costs twice the
  // shared-memory reads, so not sooner).
  const long long big = (long long)((g.M + 127) / 128) * ((g.N + 127) / 128) * g.nz;
  if (big < num_sms) return launch_gemm_simt_tile<Epi, 4, 4>(g, op, ep, stream);
  // Chains of different length (1 to L segments) end more evenly in half tiles while there are only a few tiles per SM:
  // feature gradient of the 12-layer, 1024-feature, 512-token step 1700 -> 1556 us.  Equal chains lose 10 % by them.
  if (g.mode == kDecDFeat && g.L > 1 && big < 8 * num_sms) return launch_gemm_simt_tile<Epi, 8, 4>(g, op, ep, stream);
  return launch_gemm_simt_tile<Epi, 8, 8>(g, op, ep, stream);
}

}  // namespace clt
