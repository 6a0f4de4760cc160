// C entry points of the dense contractions.  Each builds the slab geometry and the
// operand descriptions and dispatches to the fp32 CUDA-core kernel (bf16 == 0) or the
// bf16 tcgen05 kernel (bf16 == 1) with the epilogue that fuses the rest of the op.
#include "../../include/clt_b200.h"
#include "epilogues.cuh"
#include "gemm_simt.cuh"
#include "gemm_tc.cuh"
#include "kernels.h"

using namespace clt;
typedef __nv_bfloat16 bf16_t;

namespace {

// One stacked operand described once for both kernels.
//   k_contig = 1: matrix z is [rows_mn, K] with K contiguous   (K-major)
//   k_contig = 0: matrix z is [K, rows_mn] with MN contiguous  (MN-major)
struct Operand {
  const void* ptr;
  int k_contig;
  long long mn, k, z_count;
};

tc::TcOperand tc_operand(const Operand& o) {
  tc::TcOperand t;
  t.ptr = o.ptr;
  t.mn_major = o.k_contig ? 0 : 1;
  t.inner = o.k_contig ? o.k : o.mn;
  t.rows = o.k_contig ? o.mn : o.k;
  t.row_stride = t.inner;
  t.z_count = o.z_count;
  t.z_stride = o.mn * o.k;
  return t;
}

SimtOperands simt_operands(const Operand& a, const Operand& b) {
  SimtOperands s{};
  s.A = (const float*)a.ptr;
  s.B = (const float*)b.ptr;
  s.sAz = a.mn * a.k;
  s.sAm = a.k_contig ? a.k : 1;
  s.sAk = a.k_contig ? 1 : a.mn;
  s.sBz = b.mn * b.k;
  s.sBn = b.k_contig ? b.k : 1;
  s.sBk = b.k_contig ? 1 : b.mn;
  return s;
}

// A_MN / B_MN: the operand is MN-major (k_contig == 0), fixed by the op and so by the instantiation
template <class EpiF32, class EpiBf16, bool A_MN, bool B_MN>
int run_gemm(const GemmGeom& g, const Operand& a, const Operand& b, const typename EpiF32::Params& p32,
             const typename EpiBf16::Params& p16, int bf16, int* status, cudaStream_t stream) {
  if (bf16) {
    CLT_CHECK_ARG(status != nullptr, "the tensor-core path needs a device status word");
    CLT_CHECK_ARG(a.k_contig == (A_MN ? 0 : 1) && b.k_contig == (B_MN ? 0 : 1), "gemm: operand layout");
    return tc::launch_gemm_tc<EpiBf16, A_MN, B_MN>(g, tc_operand(a), tc_operand(b), p16, status, device_sm_count(),
                                                   stream);
  }
  return launch_gemm_simt<EpiF32>(g, simt_operands(a, b), p32, device_sm_count(), stream);
}

bool dims_ok(int B, int L, int D, int F) { return B > 0 && L > 0 && D > 0 && F > 0; }

// Cuts the decoder's contraction axis into parts (gemm.cuh) where that is faster; sets g.kb_per_part and returns the
// number of parts, or 0 for whole chains.
//
// Output tiles run `slots` at a time (one to an SM in bf16, two in fp32), so a fair share of the work is
// total * tiles / slots k-blocks, and the launch lasts as long as its longest chain.  Parts come into question when
// that chain is over 3/2 of the share: at 1.37 (12 layers x 9 tiles on 148 SMs, 384 blocks each) whole chains took 170
// us and parts 200 us.  Parts of half a share keep the last wave short; below 8 blocks a part's output costs more than its
// products.  Then both forms are estimated (us):
//   * a bf16 block takes its CTA 0.39 (staging its operands from L2), whatever the tile is filled with;
//   * fp32: 2.2 in a 128 x 128 tile, two to an SM, 0.62 of the SM's time in a 64 x 64 tile but 0.9 of its own; small
//     tiles are what whole chains get when the large ones are fewer than the SMs, and what parts often do not get;
//   * the weights cross HBM once at 5.5 TB/s;
//   * parts add a launch and their sums' way to memory and back: 6 us and 8 bytes each at 5 TB/s.
// 430 random sizes of 5 to 1500 tokens, 64 to 2304 wide, whole -> parts: 9 tiles with chains of 157 to 1884 blocks (12
// calls) 4604 -> 568 us, fp32 24 tiles of 1 to 12 segments 1784 -> 1460; none that is taken is slower by more than
// 2 %, and none that is left whole would have gained more than a fifth.  By the 3/2 alone over a dozen lost 10 to 50 %
// (short chains over many tokens: 8 layers x 528 tokens x 512 wide, 35 blocks 29.6 -> 44.0 us; few tokens in fp32:
// 8 x 43 x 2296, 591 blocks 716 -> 976 us).
//
// Parts are also the more exact form, since accumulators take fewer terms.  Relative error against float64 over 24
// sizes of these ranges, whole -> parts: 1.3e-4 -> 2.6e-6 (bf16, 120000 features), 8.3e-6 -> 2.7e-7 (10000), 5 to 80
// times less in bf16 and 2 to 6 times less in fp32, nowhere more.  In bf16 the error goes with a part's length (the
// tensor-core accumulator truncates), and half a share is the longest that is taken: 257 tokens, 120000 features, 768 wide,
// 33 parts of 58 blocks 2.9e-6 and 76 us; 16 of 119, which fill one round of the chip, would be 68 us and 6.6e-6; 49 of 39,
// which fill three, 80 us and 1.8e-6.
int plan_parts(GemmGeom& g, bool bf16, int sms) {
  const auto up = [](long long a, long long b) { return (a + b - 1) / b; };
  const int kb = bf16 ? tc::kBK : kSimtBK, kb_per_seg = (int)up(g.Kseg, kb);
  const long long tiles = up(g.M, 128) * up(g.N, bf16 ? tc::kBN : 128), slots = bf16 ? sms : 2 * sms;
  long long total = 0, longest = 0;
  for (int z = 0; z < g.nz; ++z) {
    const long long n = (long long)seg_count(g, z) * kb_per_seg;
    total += n;
    longest = n > longest ? n : longest;
  }
  if (longest < 32 || longest * slots * 2 <= total * tiles * 3) return 0;
  const long long half = up(total * tiles, 2 * slots), part = half < 8 ? 8 : half;
  g.kb_per_part = (int)part;
  long long parts = 0;
  for (int z = 0; z < g.nz; ++z) parts += part_count(g, z, kb_per_seg);
  double whole, split;
  if (bf16) {
    whole = 0.39 * longest;
    split = 0.39 * part * up(parts * tiles, slots);
  } else {
    const long long small = up(g.M, 64) * up(g.N, 64);
    whole = tiles * g.nz < sms ? fmax(0.9 * longest, 0.62 * total * small / sms) : 2.2 * longest;
    split = parts * tiles < sms ? part * fmax(0.9, 0.62 * up(parts * small, sms))
                                : 2.2 * part * up(parts * tiles, slots);
  }
  const double weights = (double)total * kb * g.N * (bf16 ? 2 : 4) / 5.5e6;
  split = fmax(split, weights) + 6.0 + 8.0 * parts * g.M * g.N / 5e6;
  if (parts > 65535 || 1.05 * split >= fmax(whole, weights)) return g.kb_per_part = 0;
  return (int)parts;
}

GemmGeom decoder_geom(int B, int L, int D, int F, int crosslayer) {
  return GemmGeom{crosslayer ? kDecFwd : kBatched, B, D, F, L, L};
}

// recon[b, t, d] = b_dec[t, d] + the partial sums of target t's parts, in their order.  V consecutive d per thread.
template <int V>
__global__ void __launch_bounds__(256) sum_parts_kernel(const float* __restrict__ ws, const float* __restrict__ b_dec,
                                                        float* __restrict__ recon, GemmGeom g, int kb_per_seg) {
  const int t = blockIdx.y;
  const long long i = (blockIdx.x * 256ll + threadIdx.x) * V;
  const long long slab = (long long)g.M * g.N;
  if (i >= slab) return;
  int first = 0;
  for (int u = 0; u < t; ++u) first += part_count(g, u, kb_per_seg);
  const int n = part_count(g, t, kb_per_seg);
  const long long b = i / g.N;
  const int d = (int)(i - b * g.N);
  const float* p = ws + first * slab + i;
  float acc[V];
#pragma unroll
  for (int q = 0; q < V; ++q) acc[q] = b_dec != nullptr ? __ldg(b_dec + (size_t)t * g.N + d + q) : 0.f;
#pragma unroll 8
  for (int j = 0; j < n; ++j) {
    if (V == 4) {
      const float4 v = __ldcs(reinterpret_cast<const float4*>(p + j * slab));
      acc[0] += v.x, acc[1 % V] += v.y, acc[2 % V] += v.z, acc[3 % V] += v.w;
    } else {
      acc[0] += __ldcs(p + j * slab);
    }
  }
  float* o = recon + ((size_t)b * gridDim.y + t) * g.N + d;
  if (V == 4)
    *reinterpret_cast<float4*>(o) = make_float4(acc[0], acc[1 % V], acc[2 % V], acc[3 % V]);
  else
    *o = acc[0];
}

}  // namespace

extern "C" {

int clt_encoder_fwd_act(const void* xn, const void* W_enc, const float* b_enc, const float* theta,
                        const float* dec_norm, void* z_out, void* feat_out, uint32_t* fired_bits, float* loss_acc,
                        float c_sparsity, int use_tanh, int want_pre, int B, int L, int D, int F, int bf16,
                        int* status, clt_stream_t stream) {
  CLT_CHECK_ARG(dims_ok(B, L, D, F), "encoder_fwd_act: bad dims B=%d L=%d D=%d F=%d", B, L, D, F);
  CLT_CHECK_ARG(xn && W_enc && b_enc && z_out && feat_out && loss_acc, "encoder_fwd_act: null pointer");
  GemmGeom g{kBatched, B, F, D, L, L};
  Operand a{xn, 1, B, D, L}, b{W_enc, 0, F, D, L};
  epi::EncJumpReLU<float>::Params p32{b_enc, theta, dec_norm, (float*)z_out, (float*)feat_out, fired_bits, loss_acc,
                                      c_sparsity, use_tanh, want_pre};
  epi::EncJumpReLU<bf16_t>::Params p16{b_enc, theta, dec_norm, (bf16_t*)z_out, (bf16_t*)feat_out, fired_bits,
                                       loss_acc, c_sparsity, use_tanh, want_pre};
  return run_gemm<epi::EncJumpReLU<float>, epi::EncJumpReLU<bf16_t>, false, true>(g, a, b, p32, p16, bf16, status,
                                                                      (cudaStream_t)stream);
}

int clt_encoder_fwd_store(const void* xn, const void* W_enc, void* z_out, int B, int L, int D, int F, int bf16,
                          int* status, clt_stream_t stream) {
  CLT_CHECK_ARG(dims_ok(B, L, D, F), "encoder_fwd_store: bad dims B=%d L=%d D=%d F=%d", B, L, D, F);
  CLT_CHECK_ARG(xn && W_enc && z_out, "encoder_fwd_store: null pointer");
  GemmGeom g{kBatched, B, F, D, L, L};
  Operand a{xn, 1, B, D, L}, b{W_enc, 0, F, D, L};
  epi::StoreZ<float>::Params p32{(float*)z_out};
  epi::StoreZ<bf16_t>::Params p16{(bf16_t*)z_out};
  return run_gemm<epi::StoreZ<float>, epi::StoreZ<bf16_t>, false, true>(g, a, b, p32, p16, bf16, status,
                                                                        (cudaStream_t)stream);
}

int clt_encoder_layer_fwd(const void* x, int in_dtype, const void* W_enc, const float* b_enc, void* xn, float* out, int B,
                          int D, int F, int* status, clt_stream_t stream) {
  CLT_CHECK_ARG(dims_ok(B, 1, D, F), "encoder_layer_fwd: bad dims B=%d D=%d F=%d", B, D, F);
  CLT_CHECK_ARG(x && W_enc && xn && out && status, "encoder_layer_fwd: null pointer");
  CLT_CHECK_ARG((uintptr_t)out % 16 == 0, "encoder_layer_fwd: out must be 16-byte aligned");
  if (int rc = prep_input(x, in_dtype, nullptr, nullptr, xn, 1, B, 1, D, 1, (cudaStream_t)stream)) return rc;
  GemmGeom g{kBatched, B, F, D, 1, 1};
  Operand a{xn, 1, B, D, 1}, b{W_enc, 0, F, D, 1};
  epi::PreOut<bf16_t>::Params p{out, b_enc};
  return tc::launch_gemm_tc<epi::PreOut<bf16_t>, false, true>(g, tc_operand(a), tc_operand(b), p, status,
                                                              device_sm_count(), (cudaStream_t)stream);
}

int clt_decoder_layer_fwd(const float* x, int64_t ld, const void* W_dec, const float* b_dec, void* feat, float* recon,
                          float* ws, int64_t ws_floats, int B, int K, int D, int bf16, int* status,
                          clt_stream_t stream) {
  if (int rc = clt_import_rows(x, ld, feat, B, K, bf16, stream)) return rc;
  return clt_decoder_dense_fwd_ws(feat, W_dec, b_dec, recon, ws, ws_floats, B, 1, D, K, 0, bf16, status, stream);
}

int clt_decoder_dense_fwd(const void* feat, const void* W_dec, const float* b_dec, float* recon, int B, int L, int D,
                          int F, int crosslayer, int bf16, int* status, clt_stream_t stream) {
  return clt_decoder_dense_fwd_ws(feat, W_dec, b_dec, recon, nullptr, 0, B, L, D, F, crosslayer, bf16, status, stream);
}

int clt_decoder_dense_fwd_ws(const void* feat, const void* W_dec, const float* b_dec, float* recon, float* ws,
                             int64_t ws_floats, int B, int L, int D, int F, int crosslayer, int bf16, int* status,
                             clt_stream_t stream) {
  CLT_CHECK_ARG(dims_ok(B, L, D, F), "decoder_dense_fwd: bad dims B=%d L=%d D=%d F=%d", B, L, D, F);
  CLT_CHECK_ARG(feat && W_dec && recon, "decoder_dense_fwd: null pointer");
  const int P = crosslayer ? L * (L + 1) / 2 : L;
  GemmGeom g = decoder_geom(B, L, D, F, crosslayer);
  Operand a{feat, 1, B, F, L}, b{W_dec, 0, D, F, P};
  if (ws != nullptr) {
    CLT_CHECK_ARG((uintptr_t)ws % 16 == 0, "decoder_dense_fwd: the workspace must be 16-byte aligned");
    const long long slab = (long long)B * D;
    const int parts = plan_parts(g, bf16 != 0, device_sm_count());
    if (parts > 0 && parts * slab <= ws_floats) {
      g.nz = parts;
      epi::DecOut::Params pp{ws, nullptr, (long long)D, slab};
      if (int rc = run_gemm<epi::DecOut, epi::DecOut, false, true>(g, a, b, pp, pp, bf16, status, (cudaStream_t)stream))
        return rc;
      const int kb = bf16 ? tc::kBK : kSimtBK, kb_per_seg = (F + kb - 1) / kb;
      if (D % 4 == 0 && ((uintptr_t)recon | (uintptr_t)b_dec) % 16 == 0) {
        sum_parts_kernel<4><<<dim3((unsigned)((slab / 4 + 255) / 256), L), 256, 0, (cudaStream_t)stream>>>(
            ws, b_dec, recon, g, kb_per_seg);
      } else {
        sum_parts_kernel<1><<<dim3((unsigned)((slab + 255) / 256), L), 256, 0, (cudaStream_t)stream>>>(
            ws, b_dec, recon, g, kb_per_seg);
      }
      CLT_CHECK_CUDA(cudaGetLastError());
      return 0;
    }
    g.kb_per_part = 0;  // the workspace is too small: whole chains
  }
  epi::DecOut::Params p{recon, b_dec, (long long)L * D, (long long)D};
  return run_gemm<epi::DecOut, epi::DecOut, false, true>(g, a, b, p, p, bf16, status, (cudaStream_t)stream);
}

int clt_decoder_dense_parts(int B, int L, int D, int F, int crosslayer, int bf16, int num_sms) {
  if (!dims_ok(B, L, D, F)) return 0;
  GemmGeom g = decoder_geom(B, L, D, F, crosslayer);
  return plan_parts(g, bf16 != 0, num_sms > 0 ? num_sms : device_sm_count());
}

int clt_decoder_dense_fwd_push(const void* feat, const void* W_dec, const float* b_dec, const uint64_t* rank_bases,
                               int rows_per_rank, int n_ranks, int my_slot, int slot_bf16, int B, int L, int D, int F,
                               int crosslayer, int bf16, int* status, clt_stream_t stream) {
  CLT_CHECK_ARG(dims_ok(B, L, D, F), "decoder_dense_fwd_push: bad dims B=%d L=%d D=%d F=%d", B, L, D, F);
  CLT_CHECK_ARG(feat && W_dec && rank_bases, "decoder_dense_fwd_push: null pointer");
  CLT_CHECK_ARG(n_ranks > 0 && n_ranks <= epi::kMaxPushRanks && rows_per_rank > 0 &&
                    (long long)rows_per_rank * n_ranks >= B,
                "decoder_dense_fwd_push: %d ranks x %d rows do not cover B=%d (at most %d ranks)", n_ranks,
                rows_per_rank, B, epi::kMaxPushRanks);
  const int P = crosslayer ? L * (L + 1) / 2 : L;
  GemmGeom g{crosslayer ? kDecFwd : kBatched, B, D, F, L, L};
  Operand a{feat, 1, B, F, L}, b{W_dec, 0, D, F, P};
  epi::DecOutPush::Params p;
  for (int r = 0; r < epi::kMaxPushRanks; ++r) p.bases[r] = r < n_ranks ? (unsigned long long)rank_bases[r] : 0ull;
  p.bias = b_dec;
  p.rows_per_rank = rows_per_rank;
  CLT_CHECK_ARG(my_slot >= 0 && my_slot < n_ranks, "decoder_dense_fwd_push: slot %d of %d", my_slot, n_ranks);
  p.ld = (long long)L * D;
  p.zstride = (long long)D;
  p.slot_offset = (long long)my_slot * rows_per_rank * L * D;
  p.slot_bf16 = slot_bf16 ? 1 : 0;
  return run_gemm<epi::DecOutPush, epi::DecOutPush, false, true>(g, a, b, p, p, bf16, status, (cudaStream_t)stream);
}

int clt_decoder_dense_bwd_dfeat(const void* drecon, const void* W_dec, const void* z_in, const float* b_enc,
                                const float* theta, const float* dec_norm, void* dpre_out, float* dtheta, float* dbenc,
                                float* dnorm, float bandwidth, float lam, float c_sparsity, float pal, int use_tanh,
                                const float* gscale, int B, int L, int D, int F, int crosslayer, int bf16, int* status,
                                clt_stream_t stream) {
  CLT_CHECK_ARG(dims_ok(B, L, D, F), "decoder_dense_bwd_dfeat: bad dims B=%d L=%d D=%d F=%d", B, L, D, F);
  CLT_CHECK_ARG(drecon && W_dec && z_in && b_enc && dpre_out && dbenc, "decoder_dense_bwd_dfeat: null pointer");
  CLT_CHECK_ARG(bandwidth > 0.f, "decoder_dense_bwd_dfeat: bandwidth must be positive");
  const int P = crosslayer ? L * (L + 1) / 2 : L;
  GemmGeom g{crosslayer ? kDecDFeat : kBatched, B, F, D, L, L};
  // A: drecon[t] as [B, D] (K = D contiguous); B: W_dec[p] as [F (N), D (K)], K contiguous
  Operand a{drecon, 1, B, D, L}, b{W_dec, 1, F, D, P};
  epi::DFeatJumpReLU<float>::Params p32{(const float*)z_in, b_enc, theta, dec_norm, (float*)dpre_out, dtheta, dbenc,
                                        dnorm, bandwidth, lam, c_sparsity, pal, use_tanh, gscale};
  epi::DFeatJumpReLU<bf16_t>::Params p16{(const bf16_t*)z_in, b_enc, theta, dec_norm, (bf16_t*)dpre_out, dtheta, dbenc,
                                         dnorm, bandwidth, lam, c_sparsity, pal, use_tanh, gscale};
  return run_gemm<epi::DFeatJumpReLU<float>, epi::DFeatJumpReLU<bf16_t>, false, false>(g, a, b, p32, p16, bf16, status,
                                                                          (cudaStream_t)stream);
}

int clt_decoder_dense_bwd_dfeat_raw(const void* drecon, const void* W_dec, void* g_out, int B, int L, int D, int F,
                                    int crosslayer, int bf16, int* status, clt_stream_t stream) {
  CLT_CHECK_ARG(dims_ok(B, L, D, F), "decoder_dense_bwd_dfeat_raw: bad dims B=%d L=%d D=%d F=%d", B, L, D, F);
  CLT_CHECK_ARG(drecon && W_dec && g_out, "decoder_dense_bwd_dfeat_raw: null pointer");
  const int P = crosslayer ? L * (L + 1) / 2 : L;
  GemmGeom g{crosslayer ? kDecDFeat : kBatched, B, F, D, L, L};
  Operand a{drecon, 1, B, D, L}, b{W_dec, 1, F, D, P};
  epi::StoreZ<float>::Params p32{(float*)g_out};
  epi::StoreZ<bf16_t>::Params p16{(bf16_t*)g_out};
  return run_gemm<epi::StoreZ<float>, epi::StoreZ<bf16_t>, false, false>(g, a, b, p32, p16, bf16, status,
                                                                         (cudaStream_t)stream);
}

int clt_decoder_dense_bwd_dw(const void* feat, const void* drecon, float* dW, const float* rowcoef,
                             const float* W_master, int B, int L, int D, int F, int crosslayer, int bf16, int* status,
                             clt_stream_t stream) {
  CLT_CHECK_ARG(dims_ok(B, L, D, F), "decoder_dense_bwd_dw: bad dims B=%d L=%d D=%d F=%d", B, L, D, F);
  CLT_CHECK_ARG(feat && drecon && dW, "decoder_dense_bwd_dw: null pointer");
  CLT_CHECK_ARG(rowcoef == nullptr || W_master != nullptr, "decoder_dense_bwd_dw: rowcoef needs the master weights");
  const int P = crosslayer ? L * (L + 1) / 2 : L;
  GemmGeom g{crosslayer ? kDecDW : kBatched, F, D, B, L, P};
  // A: feat[s]^T, stored [B (K), F (M)] with M contiguous; B: drecon[t], stored [B (K), D (N)] with N contiguous
  Operand a{feat, 0, F, B, L}, b{drecon, 0, D, B, L};
  epi::GradOut::Params p{dW, rowcoef, W_master, crosslayer ? 1 : 0};
  return run_gemm<epi::GradOut, epi::GradOut, true, true>(g, a, b, p, p, bf16, status, (cudaStream_t)stream);
}

int clt_encoder_dense_bwd_dw(const void* xn, const void* dpre, float* dW, int B, int L, int D, int F, int bf16,
                             int* status, clt_stream_t stream) {
  CLT_CHECK_ARG(dims_ok(B, L, D, F), "encoder_dense_bwd_dw: bad dims B=%d L=%d D=%d F=%d", B, L, D, F);
  CLT_CHECK_ARG(xn && dpre && dW, "encoder_dense_bwd_dw: null pointer");
  GemmGeom g{kBatched, D, F, B, L, L};
  Operand a{xn, 0, D, B, L}, b{dpre, 0, F, B, L};
  epi::GradOut::Params p{dW, nullptr, nullptr, 0};
  return run_gemm<epi::GradOut, epi::GradOut, true, true>(g, a, b, p, p, bf16, status, (cudaStream_t)stream);
}

}  // extern "C"
