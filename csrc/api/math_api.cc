// C entry points of the element-wise passes (kernels/fused_math.cu).  The reference has no counterpart.
#include <cuda_runtime.h>

#include <cmath>
#include <initializer_list>

#include "../comm/comm.h"
#include "../core/log.h"
#include "../include/nccl.h"
#include "../kernels/fused_math.h"
#include "../kernels/launch.h"

using namespace amem;

namespace {

inline ncclResult_t R(Status s) {
  if (s != kSuccess) LOGW("%s: %s", status_name(s), last_error_slot().c_str());
  return (ncclResult_t)s;
}

bool aligned16(const void* a, const void* b, const void* c) { return !(((uintptr_t)a | (uintptr_t)b | (uintptr_t)c) & 15); }

// (an empty tensor has no address: asked only where there is something to read)
bool missing(std::initializer_list<const void*> buffers) {
  for (const void* p : buffers)
    if (!p) return true;
  return false;
}

}  // namespace

extern "C" {

ncclResult_t amemSwiGLU(const void* gate, const void* up, long long ld, void* act, long long rows, int F, cudaStream_t stream) {
  if (rows < 0 || F <= 0 || F % 8 || ld < F || ld % 8 || !aligned16(gate, up, act))
    return R(fail(kInvalidArgument, "amemSwiGLU: rows=%lld F=%d ld=%lld (multiples of 8, 16-byte aligned)", rows, F, ld));
  if (rows > 0 && missing({gate, up, act})) return R(fail(kInvalidArgument, "amemSwiGLU: null buffer"));
  return rows == 0 ? ncclSuccess : R(launch_swiglu(gate, up, (long)ld, act, (long)rows, F, stream));
}

ncclResult_t amemSwiGLUGrad(const void* gate, const void* up, long long ld, const void* g_act, void* g_gate, void* g_up, long long rows, int F,
                            cudaStream_t stream) {
  if (rows < 0 || F <= 0 || F % 8 || ld < F || ld % 8 || !aligned16(gate, up, g_act) || !aligned16(g_gate, g_up, nullptr))
    return R(fail(kInvalidArgument, "amemSwiGLUGrad: rows=%lld F=%d ld=%lld (multiples of 8, 16-byte aligned)", rows, F, ld));
  if (rows > 0 && missing({gate, up, g_act, g_gate, g_up})) return R(fail(kInvalidArgument, "amemSwiGLUGrad: null buffer"));
  return rows == 0 ? ncclSuccess : R(launch_swiglu_grad(gate, up, (long)ld, g_act, g_gate, g_up, (long)rows, F, stream));
}

ncclResult_t amemRmsNorm(const void* x, const void* w, void* y, float* rstd, long long rows, int dim, double eps, cudaStream_t stream) {
  if (!rms_norm_takes((long)rows, dim) || !aligned16(x, w, y) || missing({x, w, y}))
    return R(fail(kInvalidArgument, "amemRmsNorm: rows=%lld dim=%d (a multiple of 8 up to 16384, 16-byte aligned)", rows, dim));
  return R(launch_rms_norm(x, w, y, rstd, (long)rows, dim, (float)eps, stream));
}

int amemRmsNormGradBlocks(long long rows) { return rms_norm_grad_blocks((long)rows); }

ncclResult_t amemRmsNormGrad(const void* g_y, const void* x, const void* w, const float* rstd, void* g_x, float* part_w, void* g_w, long long rows, int dim,
                             cudaStream_t stream) {
  if (!rms_norm_takes((long)rows, dim) || !aligned16(g_y, x, w) || !aligned16(g_x, part_w, nullptr) || missing({g_y, x, w, rstd}) || (g_w && !part_w))
    return R(fail(kInvalidArgument, "amemRmsNormGrad: rows=%lld dim=%d (a multiple of 8 up to 16384, 16-byte aligned)", rows, dim));
  return R(launch_rms_norm_grad(g_y, x, w, rstd, g_x, part_w, g_w, (long)rows, dim, stream));
}

ncclResult_t amemEmbeddingGradShared(const void* g, const long long* ids, void* g_table, void* work, int tokens, int dim, long long rows, cudaStream_t stream) {
  if (tokens <= 0 || dim <= 0 || dim % 8 || rows <= 0 || missing({g, ids, g_table, work}) || !aligned16(g, g_table, work))
    return R(fail(kInvalidArgument, "amemEmbeddingGrad: tokens=%d dim=%d (a multiple of 8) rows=%lld, 16-byte aligned", tokens, dim, rows));
  return R(launch_embedding_grad(g, ids, g_table, (unsigned char*)work, tokens, dim, rows, stream));
}

ncclResult_t amemEmbeddingGrad(const void* g, const long long* ids, void* g_table, int tokens, int dim, long long rows, cudaStream_t stream) {
  void* work = nullptr;
  if (tokens > 0 && !missing({g, ids, g_table})) {
    const cudaError_t e = cudaMallocAsync(&work, ((size_t)tokens + 15) / 16 * 16, stream);
    if (e != cudaSuccess) return R(fail(kCudaError, "amemEmbeddingGrad: %s", cudaGetErrorString(e)));
  }
  const ncclResult_t r = amemEmbeddingGradShared(g, ids, g_table, work, tokens, dim, rows, stream);
  if (work) cudaFreeAsync(work, stream);
  return r;
}

ncclResult_t amemRotate(const void* const* in, void* const* out, const int* heads, const long long* strides, int tensors, const float* cos, const float* sin,
                        int batch, int seq, int dim, int inverse, cudaStream_t stream) {
  if (tensors < 1 || tensors > 2 || batch <= 0 || seq <= 0 || (long long)batch * seq > 0x7fffffffLL || dim <= 0 || dim % 8 || missing({in, out, heads, strides}) ||
      missing({cos, sin}) || !aligned16(cos, sin, nullptr))
    return R(fail(kInvalidArgument, "amemRotate: tensors=%d batch=%d seq=%d dim=%d (a multiple of 8)", tensors, batch, seq, dim));
  Rotation a = {};
  for (int i = 0; i < tensors; ++i) {
    const long long* st = strides + 6 * i;
    bool fits = heads[i] > 0 && (long long)heads[i] * dim <= 0x3fffffffLL && !missing({in[i], out[i]}) && aligned16(in[i], out[i], nullptr);
    for (int j = 0; j < 6; ++j) fits = fits && st[j] >= 0 && st[j] % 8 == 0;
    if (!fits) return R(fail(kInvalidArgument, "amemRotate: tensor %d needs heads, 16-byte aligned rows and strides that are multiples of 8", i));
    a.t[i] = {(const char*)in[i], (char*)out[i], heads[i], (long)st[0], (long)st[1], (long)st[2], (long)st[3], (long)st[4], (long)st[5]};
  }
  a.cos = cos;
  a.sin = sin;
  a.seq = seq;
  a.vecs = dim / 8;
  a.turn = inverse ? -1.f : 1.f;
  return R(launch_rotate(a, batch, stream));
}

static Status sum_pieces(const char* what, const void* const* src, float* const* dst, const long long* n, int pieces, double scale, int block_cap,
                         cudaStream_t stream) {
  if (pieces < 0 || (pieces > 0 && missing({src, dst, n}))) return fail(kInvalidArgument, "%s: %d pieces", what, pieces);
  for (int i = 0; i < pieces; ++i) {
    if (n[i] < 0 || (n[i] > 0 && missing({src[i], dst[i]})) || ((uintptr_t)src[i] & 1) || ((uintptr_t)dst[i] & 3))
      return fail(kInvalidArgument, "%s: piece %d of %lld elements", what, i, n[i]);
  }
  return launch_sum_pieces(src, dst, n, pieces, (float)scale, block_cap, stream);
}

ncclResult_t amemSumPieces(const void* const* src, float* const* dst, const long long* n, int pieces, double scale, cudaStream_t stream) {
  return R(sum_pieces("amemSumPieces", src, dst, n, pieces, scale, 0, stream));
}

ncclResult_t amemSumPiecesLocal(const void* const* src, float* const* dst, const long long* n, int pieces, double scale, ncclComm_t comm, cudaStream_t stream) {
  if (!comm) return ncclInvalidArgument;
  Comm* c = reinterpret_cast<Comm*>(comm);
  Status s = c->check_usable("amemSumPiecesLocal");
  if (s == kSuccess && c->nranks() != 1) s = fail(kInvalidArgument, "amemSumPiecesLocal: a communicator of one rank expected");
  if (s == kSuccess) s = c->prepare_stream(stream);
  return R(s == kSuccess ? sum_pieces("amemSumPiecesLocal", src, dst, n, pieces, scale, c->block_cap(), stream) : s);
}

ncclResult_t amemSumPiecesPlan(const long long* n, int pieces, int block_cap, size_t* blocks) {
  if (!blocks || pieces < 0 || (pieces > 0 && !n)) return ncclInvalidArgument;
  *blocks = sum_pieces_blocks(n, pieces, block_cap);
  return ncclSuccess;
}

ncclResult_t amemAdamW(const float* grad, float* m, float* v, float* master, void* shard_bf16, long long n, double lr, double beta1, double beta2,
                       double eps, double weight_decay, long long step, cudaStream_t stream) {
  if (n < 0 || step < 1 || !aligned16(grad, m, v) || !aligned16(master, shard_bf16, nullptr))
    return R(fail(kInvalidArgument, "amemAdamW: n=%lld step=%lld (buffers 16-byte aligned)", n, step));
  if (n == 0) return ncclSuccess;
  if (missing({grad, m, v, master, shard_bf16})) return R(fail(kInvalidArgument, "amemAdamW: null buffer"));
  AdamW a;
  a.lr = (float)lr;
  a.b1 = (float)beta1;
  a.one_minus_b1 = (float)(1.0 - beta1);
  a.b2 = (float)beta2;
  a.one_minus_b2 = (float)(1.0 - beta2);
  a.c1 = (float)(1.0 - std::pow(beta1, (double)step));
  a.c2 = (float)(1.0 - std::pow(beta2, (double)step));
  a.eps = (float)eps;
  a.decay = (float)(1.0 - lr * weight_decay);
  return R(launch_adamw(grad, m, v, master, shard_bf16, (long)n, a, stream));
}

}  // extern "C"
