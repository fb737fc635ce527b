// The launches of one transformer block, forward and backward, issued by one call each.
//
// A block is nine kernels forward and about twenty backward. Issued one by one from Python, each costs 20 us of interpreter, autograd and
// binding, which is more than most of them take below a few thousand tokens: the 64 M decoder at 3 x 1001 tokens was held to 9.7 ms a
// step by a host that had 5.3 ms of kernels to launch. Here the same kernels, with the same arguments in the same order, are launched
// from C at 3 us each. Nothing is kept between calls; all memory is the caller's.
#include "sm100_common.cuh"
#include "inv_api.h"

extern "C" {
int inv_norm_fwd(const void* x, const void* res, const void* gamma, const void* beta, void* y, void* xsum, float* mean, float* rstd, int T, int D,
                 float eps, int rms, void* stream);
int inv_norm_bwd_grid(int T);
int inv_norm_bwd(const void* dy, const void* x, const void* gamma, const float* mean, const float* rstd, const void* dres, void* dx, float* dgamma,
                 float* dbeta, float* scratch, int T, int D, int rms, void* stream);
int inv_norm_bwd_colsum(const void* dy, const void* x, const void* gamma, const float* mean, const float* rstd, const void* dres, void* dx,
                        float* dgamma, float* dbeta, float* colsum, float* scratch, int T, int D, int rms, void* stream);
int inv_colsum(const void* x, float* out, int T, int N, int ld, void* stream);
int inv_act(const void* x, const void* dy, void* out, long rows, int F, int mode, void* stream);
int inv_rope(void* buf, const int* pos, const float* cos_t, const float* sin_t, int T, int S, int ld, int col0, int nheads, int hd, int inverse,
             void* stream);
int inv_flash_attn_fwd(const void* q, const void* k, const void* v, void* out, float* lse, int B, int S, int H, int Hkv, int head_dim, int ld_q,
                       int ld_k, int ld_v, int ld_o, float scale, int causal, int window, int* status, void* stream);
long inv_flash_attn_bwd_scratch_bytes(int B, int S, int H, int head_dim);
int inv_flash_attn_bwd(const void* q, const void* k, const void* v, const void* o, const void* d_o, const float* lse, void* dq, void* dk, void* dv,
                       void* scratch, int B, int S, int H, int Hkv, int head_dim, int ld_q, int ld_k, int ld_v, int ld_o, int ld_do, int ld_dq,
                       int ld_dk, int ld_dv, float scale, int causal, int window, int* status, void* stream);
int inv_block_quant(const void* in, int in_dtype, void* out_q, int out_dtype, uint8_t* idx, float* scales, const float* codebook, int K, long n,
                    int mode, void* stream);
}

namespace inv {

__global__ void add_f32_kernel(float* __restrict__ dst, const float* __restrict__ src, int n) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) dst[i] += src[i];
}

// One block as the caller describes it (the Python side packs the same fields in the same order).
struct BlockDesc {
  // parameters, bf16; biases and beta may be null
  const void *g1, *b1, *wqkv, *bqkv, *wo, *bo, *g2, *b2, *w1, *bias1, *w2, *bias2;
  const float *cos_t, *sin_t;      // rotary tables, or null
  const int* positions;            // or null
  const float* codebook;           // of the straight-through quantiser (n_codebook > 0)
  const void* x;                   // bf16 [B * S, E]
  void* y;                         // forward: the output
  void* saved;                     // what the forward pass leaves for the backward pass (layout below)
  int* status;
  void* stream;
  // backward
  const void* dy;
  void* dx;
  const float* dy_colsum;          // column sums of dy, or null
  float* dx_colsum;                // E <= 1024: receives those of dx
  float *dg1, *db1, *dwqkv, *dbqkv, *dwo, *dbo, *dg2, *db2, *dw1, *dbias1, *dw2, *dbias2;   // fp32, added to
  void* scratch;
  long B, S, E, H, Hkv, D, F, gated, rms, n_codebook, quant_mode, quantised, kernel_select;
  long keep;                       // a backward pass follows
  double eps1, eps2, scale;
  bool in_y() const { return !keep && H * D <= E; }      // y holds what is dead before it is written
};

constexpr long AT = 256;           // every buffer starts on 256 bytes
static long up(long bytes) { return (bytes + AT - 1) / AT * AT; }

// Offsets into `saved`: the quantised weights, the activations and the statistics. Where no backward pass follows (keep = 0) buffers whose lives
// do not overlap share their place, as they do where the layers run one by one and free each result behind its last use, and what is dead before
// the last product lies in its output y: a layer of width 2048 (gated MLP of 5632, 16 heads on 4) over 16 x 4096 tokens 2.49 GB instead of 3.70.
struct BlockSaved {
  long qkv_w, o_w, w1, w2, h1, qkv, a, x2, h2, mid, act, lse, mean1, rstd1, mean2, rstd2, total;
  BlockSaved(const BlockDesc& d) {
    const long T = d.B * d.S, W = (d.H + 2 * d.Hkv) * d.D, mid_cols = d.gated ? 2 * d.F : d.F, O = d.H * d.D, q = d.quantised ? 2 : 0;
    long at = 0;
    auto take = [&](long bytes) { const long here = at; at += up(bytes); return here; };
    auto max2 = [](long a, long b) { return a > b ? a : b; };
    if (d.keep) {
      qkv_w = take(q * W * d.E); o_w = take(q * d.E * O); w1 = take(q * mid_cols * d.E); w2 = take(q * d.E * d.F);
      h1 = take(2 * T * d.E); qkv = take(2 * T * W); a = take(2 * T * O); x2 = take(2 * T * d.E); h2 = take(2 * T * d.E);
      mid = take(2 * T * mid_cols); act = take(2 * T * d.F);
      lse = take(4 * T * d.H); mean1 = take(4 * T); rstd1 = take(4 * T); mean2 = take(4 * T); rstd2 = take(4 * T);
    } else {
      qkv_w = o_w = w1 = w2 = take(q * max2(max2(W * d.E, d.E * O), max2(mid_cols * d.E, d.E * d.F)));   // each is quantised in front of its product
      h1 = a = h2 = take(d.in_y() ? 0 : 2 * T * max2(d.E, O));             // norm 1, attention, norm 2: each dead before the next is written
      const long mlp = up(2 * T * d.E) + up(2 * T * d.F) + up(2 * T * mid_cols);
      qkv = x2 = take(max2(up(2 * T * W), mlp));                           // q, k, v are dead behind attention; then x2 and the MLP's activations
      act = x2 + up(2 * T * d.E); mid = act + up(2 * T * d.F);
      lse = take(4 * T * d.H); mean1 = mean2 = take(4 * T); rstd1 = rstd2 = take(4 * T);
    }
    total = at;
  }
};
// Offsets into the backward pass's scratch. Buffers whose lives do not overlap share their place.
struct BlockScratch {
  long wide, dh, dx2, da, colsum, norm, attn, total;
  BlockScratch(const BlockDesc& d) {
    const long T = d.B * d.S, W = (d.H + 2 * d.Hkv) * d.D, mid_cols = d.gated ? 2 * d.F : d.F, O = d.H * d.D;
    long at = 0;
    auto take = [&](long bytes) { const long here = at; at += up(bytes); return here; };
    const long mlp = up(2 * T * mid_cols) + (d.gated ? up(2 * T * d.F) : 0), att = up(2 * T * W);
    wide = take(mlp > att ? mlp : att);                    // gradients of the MLP's inner activations, then of q, k and v
    dh = take(2 * T * d.E); dx2 = take(2 * T * d.E); da = take(2 * T * O); colsum = take(4 * d.E);
    norm = take((long)inv_norm_bwd_grid((int)T) * 3 * d.E * 4);
    attn = take(inv_flash_attn_bwd_scratch_bytes((int)d.B, (int)d.S, (int)d.H, (int)d.D));
    total = at;
  }
};

// The cut of a weight gradient's long reduction: tiles times cuts fill the CTA pairs twice.
static int split_k_for(long M, long N, long K) {
  const long kb = (K + 63) / 64;
  const bool pairs = M > 128 && N > 128;
  const long tiles = pairs ? ((M + 255) / 256) * ((N + 255) / 256) : ((M + 127) / 128) * ((N + 255) / 256), units = pairs ? 74 : 148;
  if (tiles >= units) return 1;
  const long cuts = 2 * units / tiles;
  return (int)(cuts < 1 ? 1 : cuts < kb ? cuts : kb);
}

struct BlockRun {
  const BlockDesc& d;
  const BlockSaved s;
  char* saved;
  int T, E, W, O, F, mid_cols, launches = 0, rc = 0;
  explicit BlockRun(const BlockDesc& desc)
      : d(desc), s(desc), saved((char*)desc.saved), T((int)(desc.B * desc.S)), E((int)desc.E), W((int)((desc.H + 2 * desc.Hkv) * desc.D)),
        O((int)(desc.H * desc.D)), F((int)desc.F), mid_cols((int)(desc.gated ? 2 * desc.F : desc.F)) {}
  void* at(long o) const { return saved + o; }
  void* early(long o) const { return d.in_y() ? (char*)d.y : saved + o; }     // norm 1, attention, norm 2 in the forward pass
  float* f32(long o) const { return (float*)(saved + o); }
  const void* weight(const void* w, long o) const { return d.quantised ? saved + o : w; }
  // runs a launch unless one before it failed
  void did(int r) {
    ++launches;
    if (rc == 0) rc = r;
  }
#define INV_RUN(call) do { if (rc == 0) did(call); } while (0)
  // C[M, N] = A[M, K] B^T; b_mn: B is stored [K, N]
  void product(const void* A, const void* B, void* C, int M, int N, int K, int b_mn, int epi, const void* bias, const void* aux_in, void* aux_out) {
    INV_RUN(inv_gemm_bf16(A, B, C, M, N, K, K, b_mn ? N : K, N, 0, b_mn, epi, bias, aux_in, aux_in || aux_out ? N : 0, aux_out, 0, 1, 1.f, d.status,
                          d.stream, (int)d.kernel_select));
  }
  // dW[N, K] += dY[T, N]^T X[T, K]
  void weight_grad(const void* dy, const void* x, float* dw, int N, int K) {
    INV_RUN(inv_gemm_bf16(dy, x, dw, N, K, T, N, K, K, 1, 1, EPI_ATOMIC, nullptr, nullptr, 0, nullptr, 1, split_k_for(N, K, T), 1.f, d.status, d.stream,
                          (int)d.kernel_select));
  }
  void bias_grad(const void* dy, const float* colsum, float* db, int N) {
    if (db == nullptr) return;
    if (colsum == nullptr) { INV_RUN(inv_colsum(dy, db, T, N, N, d.stream)); return; }
    if (rc != 0) return;
    add_f32_kernel<<<(N + 255) / 256, 256, 0, (cudaStream_t)d.stream>>>(db, colsum, N);
    const cudaError_t e = cudaGetLastError();
    did(e == cudaSuccess ? 0 : -(int)e);
  }
  void rotate(void* buf, int inverse) {
    if (d.cos_t)
      INV_RUN(inv_rope(buf, d.positions, d.cos_t, d.sin_t, T, (int)d.S, W, 0, (int)(d.H + d.Hkv), (int)d.D, inverse, d.stream));
  }
  void quantise(const void* w, long o, long n) {
    if (d.quantised)
      INV_RUN(inv_block_quant(w, 1, at(o), 1, nullptr, nullptr, d.codebook, (int)d.n_codebook, n, (int)d.quant_mode, d.stream));
  }

  void forward() {
    INV_RUN(inv_norm_fwd(d.x, nullptr, d.g1, d.b1, early(s.h1), nullptr, f32(s.mean1), f32(s.rstd1), T, E, (float)d.eps1, (int)d.rms, d.stream));
    quantise(d.wqkv, s.qkv_w, (long)W * E);
    product(early(s.h1), weight(d.wqkv, s.qkv_w), at(s.qkv), T, W, E, 0, EPI_NONE, d.bqkv, nullptr, nullptr);
    rotate(at(s.qkv), 0);
    const char* q = (const char*)at(s.qkv);
    INV_RUN(inv_flash_attn_fwd(q, q + O * 2, q + (O + d.Hkv * d.D) * 2, early(s.a), f32(s.lse), (int)d.B, (int)d.S, (int)d.H, (int)d.Hkv, (int)d.D, W, W, W, O,
                               (float)d.scale, 1, 0, d.status, d.stream));
    quantise(d.wo, s.o_w, (long)E * O);
    product(early(s.a), weight(d.wo, s.o_w), at(s.x2), T, E, O, 0, EPI_ADD, d.bo, d.x, nullptr);
    INV_RUN(inv_norm_fwd(at(s.x2), nullptr, d.g2, d.b2, early(s.h2), nullptr, f32(s.mean2), f32(s.rstd2), T, E, (float)d.eps2, (int)d.rms, d.stream));
    quantise(d.w1, s.w1, (long)mid_cols * E);
    if (d.gated) {
      product(early(s.h2), weight(d.w1, s.w1), at(s.mid), T, mid_cols, E, 0, EPI_NONE, d.bias1, nullptr, nullptr);
      INV_RUN(inv_act(at(s.mid), nullptr, at(s.act), T, F, 2, d.stream));
    } else {
      product(early(s.h2), weight(d.w1, s.w1), at(s.act), T, F, E, 0, EPI_GELU_DG, d.bias1, nullptr, at(s.mid));
    }
    quantise(d.w2, s.w2, (long)E * F);
    product(at(s.act), weight(d.w2, s.w2), d.y, T, E, F, 0, EPI_ADD, d.bias2, at(s.x2), nullptr);
  }

  void norm_backward(const void* dy, const void* x, const void* g, long mean, long rstd, const void* dres, void* dx, float* dg, float* db, float* colsum,
                     float* scratch) {
    if (E <= 1024)
      INV_RUN(inv_norm_bwd_colsum(dy, x, g, f32(mean), f32(rstd), dres, dx, dg, db, colsum, scratch, T, E, (int)d.rms, d.stream));
    else
      INV_RUN(inv_norm_bwd(dy, x, g, f32(mean), f32(rstd), dres, dx, dg, db, scratch, T, E, (int)d.rms, d.stream));
  }

  void backward() {
    const BlockScratch t(d);
    char* tmp = (char*)d.scratch;
    void *wide = tmp + t.wide, *dh = tmp + t.dh, *dx2 = tmp + t.dx2, *da = tmp + t.da;
    float *colsum = (float*)(tmp + t.colsum), *norm = (float*)(tmp + t.norm);
    // MLP
    if (d.gated) {
      void* dact = tmp + t.wide + up(2l * T * mid_cols);
      product(d.dy, weight(d.w2, s.w2), dact, T, F, E, 1, EPI_NONE, nullptr, nullptr, nullptr);
      weight_grad(d.dy, at(s.act), d.dw2, E, F);
      bias_grad(d.dy, d.dy_colsum, d.dbias2, E);
      INV_RUN(inv_act(at(s.mid), dact, wide, T, F, 3, d.stream));
    } else {
      product(d.dy, weight(d.w2, s.w2), wide, T, F, E, 1, EPI_MUL, nullptr, at(s.mid), nullptr);
      weight_grad(d.dy, at(s.act), d.dw2, E, F);
      bias_grad(d.dy, d.dy_colsum, d.dbias2, E);
    }
    product(wide, weight(d.w1, s.w1), dh, T, E, mid_cols, 1, EPI_NONE, nullptr, nullptr, nullptr);
    weight_grad(wide, at(s.h2), d.dw1, mid_cols, E);
    bias_grad(wide, nullptr, d.dbias1, mid_cols);
    norm_backward(dh, at(s.x2), d.g2, s.mean2, s.rstd2, d.dy, dx2, d.dg2, d.db2, colsum, norm);
    // attention
    product(dx2, weight(d.wo, s.o_w), da, T, O, E, 1, EPI_NONE, nullptr, nullptr, nullptr);
    weight_grad(dx2, at(s.a), d.dwo, E, O);
    bias_grad(dx2, E <= 1024 ? colsum : nullptr, d.dbo, E);
    const char* q = (const char*)at(s.qkv);
    char* dq = (char*)wide;
    INV_RUN(inv_flash_attn_bwd(q, q + O * 2, q + (O + d.Hkv * d.D) * 2, at(s.a), da, f32(s.lse), dq, dq + O * 2, dq + (O + d.Hkv * d.D) * 2, tmp + t.attn,
                               (int)d.B, (int)d.S, (int)d.H, (int)d.Hkv, (int)d.D, W, W, W, O, O, W, W, W, (float)d.scale, 1, 0, d.status, d.stream));
    rotate(dq, 1);
    product(dq, weight(d.wqkv, s.qkv_w), dh, T, E, W, 1, EPI_NONE, nullptr, nullptr, nullptr);
    weight_grad(dq, at(s.h1), d.dwqkv, W, E);
    bias_grad(dq, nullptr, d.dbqkv, W);
    norm_backward(dh, d.x, d.g1, s.mean1, s.rstd1, dx2, d.dx, d.dg1, d.db1, d.dx_colsum, norm);
  }
#undef INV_RUN
};

}  // namespace inv

using namespace inv;

// Bytes of the caller's buffer: `saved` of a forward pass that a backward pass follows (which = 0), the backward pass's scratch (1), `saved` of a
// forward pass alone (2).
extern "C" int inv_block_bytes(int which, long B, long S, long E, long H, long Hkv, long D, long F, long gated, long quantised, long* bytes) {
  if (which < 0 || which > 2 || B < 1 || S < 1 || E < 1 || H < 1 || Hkv < 1 || D < 1 || F < 1) return -ERR_BAD_ARG;
  BlockDesc d{};
  d.B = B; d.S = S; d.E = E; d.H = H; d.Hkv = Hkv; d.D = D; d.F = F; d.gated = gated; d.quantised = quantised; d.keep = which != 2;
  *bytes = which == 1 ? BlockScratch(d).total : BlockSaved(d).total;
  return 0;
}

// The cut that the products of the backward pass take (ops/gemm.py states the same rule).
extern "C" int inv_block_split_k(long M, long N, long K) { return split_k_for(M, N, K); }

// Pre-norm block: y = x2 + MLP(norm2(x2)), x2 = x + attention(norm1(x)); causal. Returns the number of launches, or a negative code.
extern "C" int inv_block_fwd(const BlockDesc* d) {
  BlockRun r(*d);
  r.forward();
  return r.rc < 0 ? r.rc : r.launches;
}

// dx and all parameter gradients (added to); `saved` as inv_block_fwd left it.
extern "C" int inv_block_bwd(const BlockDesc* d) {
  BlockRun r(*d);
  r.backward();
  return r.rc < 0 ? r.rc : r.launches;
}
