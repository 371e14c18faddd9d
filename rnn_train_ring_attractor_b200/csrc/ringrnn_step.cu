// Host-side compositions and small element-wise kernels around the operator: one call for a whole training step, the active
// columns of an action signal, decoded angles and their circular error.
#include <string.h>

#include <mutex>

#include "ringrnn_common.cuh"

namespace ringrnn {
namespace {

// ---- active columns -------------------------------------------------------------------------------------------
// One slot per call in flight: a device accumulator (zero between calls: the last block resets it) and a pinned host word
// that the last block writes.  The caller waits for the stream, so a slot is free again when the call returns.
constexpr int MASK_SLOTS = 32;
struct MaskSlot {
  unsigned long long mask;
  unsigned done, pad;
};
__device__ MaskSlot g_mask_slot[MASK_SLOTS];

__global__ void __launch_bounds__(256) active_columns_kernel(const float* __restrict__ A, size_t rows, int a_dim, int slot,
                                                             volatile unsigned long long* host) {
  __shared__ unsigned long long warp_mask[8];
  const size_t total = rows * a_dim;
  const size_t stride = (size_t)gridDim.x * blockDim.x;
  unsigned long long m = 0;
  size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x;
  int col = (int)(i % a_dim);
  const int step = (int)(stride % a_dim);
  for (; i < total; i += stride) {
    if (A[i] != 0.f) m |= 1ull << col;
    col += step;
    if (col >= a_dim) col -= a_dim;
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) m |= __shfl_xor_sync(0xffffffffu, m, o);
  if ((threadIdx.x & 31) == 0) warp_mask[threadIdx.x >> 5] = m;
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int w = 1; w < 8; ++w) m |= warp_mask[w];
    MaskSlot* s = &g_mask_slot[slot];
    if (m != 0) atomicOr(&s->mask, m);
    __threadfence();
    if (atomicAdd(&s->done, 1u) == gridDim.x - 1) {
      __threadfence();
      *host = atomicExch(&s->mask, 0ull);
      s->done = 0u;
      __threadfence_system();
    }
  }
}

std::mutex g_mask_mu;
volatile unsigned long long* g_mask_host = nullptr;  // MASK_SLOTS pinned words
unsigned g_mask_busy = 0u;                           // bit per slot

// ---- element-wise ---------------------------------------------------------------------------------------------
__device__ __forceinline__ float decode_one(float x, float y) {
  const float two_pi = 6.283185307179586f;
  const float a = fmodf(atan2f(y, x) + two_pi, two_pi);
  return a < 0.f ? a + two_pi : a;
}
__device__ __forceinline__ float circular_one(float p, float t) {
  const float two_pi = 6.283185307179586f;
  const float d = fmodf(fabsf(p - t), two_pi);
  return fminf(d, two_pi - d);
}
// four elements per thread; `vec`: both inputs and the output are 16-byte aligned.  The output may be one of the inputs.
template <class F>
__device__ __forceinline__ void map2(size_t n, bool vec, const float* a, const float* b, float* o, F f) {
  const size_t stride = (size_t)gridDim.x * blockDim.x, first = blockIdx.x * (size_t)blockDim.x + threadIdx.x;
  const size_t n4 = vec ? n / 4 : 0;
  for (size_t i = first; i < n4; i += stride) {
    const float4 x = reinterpret_cast<const float4*>(a)[i], y = reinterpret_cast<const float4*>(b)[i];
    reinterpret_cast<float4*>(o)[i] = make_float4(f(x.x, y.x), f(x.y, y.y), f(x.z, y.z), f(x.w, y.w));
  }
  for (size_t i = n4 * 4 + first; i < n; i += stride) o[i] = f(a[i], b[i]);
}
__global__ void __launch_bounds__(256) decode_angles_kernel(size_t n, bool vec, const float* x, const float* y, float* out) {
  map2(n, vec, x, y, out, [](float a, float b) { return decode_one(a, b); });
}
__global__ void __launch_bounds__(256) angular_error_kernel(size_t n, bool vec, const float* p, const float* t, float* out) {
  map2(n, vec, p, t, out, [](float a, float b) { return circular_one(a, b); });
}
bool aligned16(const void* a, const void* b, const void* c) {
  return ((reinterpret_cast<uintptr_t>(a) | reinterpret_cast<uintptr_t>(b) | reinterpret_cast<uintptr_t>(c)) & 15) == 0;
}
int grid_for(size_t n) {
  const size_t blocks = (n / 4 + 255) / 256;
  return (int)(blocks < 1 ? 1 : blocks > 148 * 16 ? 148 * 16 : blocks);
}

struct TrainLayout {
  size_t scal, red, fwd, saved, bwd, total;
};
bool train_layout(const RingRnnProblem& p, TrainLayout* l) {
  const size_t fwd = ringrnn_workspace_bytes(&p, RINGRNN_WS_FWD, 0), saved = ringrnn_workspace_bytes(&p, RINGRNN_WS_SAVED, 0),
               bwd = ringrnn_workspace_bytes(&p, RINGRNN_WS_BWD, 0);
  if (fwd == (size_t)-1 || saved == (size_t)-1 || bwd == (size_t)-1) return false;
  size_t at = 0;
  l->scal = at; at += align_up((size_t)6 * p.B * p.T * sizeof(float), 1024);
  l->red = at; at += align_up((size_t)2 * p.B * sizeof(float), 1024);
  l->saved = at; at += align_up(saved, 1024);
  // the backward starts when the forward's scratch is dead: one region serves both
  l->fwd = l->bwd = at;
  at += align_up(fwd > bwd ? fwd : bwd, 1024);
  l->total = at;
  return true;
}

}  // namespace
}  // namespace ringrnn

using namespace ringrnn;

extern "C" int ringrnn_active_columns(const float* A, long long rows, int a_dim, unsigned long long* mask, void* stream) {
  if (A == nullptr || mask == nullptr) return RINGRNN_ERR_ARG;
  if (rows <= 0 || a_dim <= 0 || a_dim > RINGRNN_MAX_ACTIVE) return RINGRNN_ERR_SHAPE;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  int slot = -1;
  {
    std::lock_guard<std::mutex> lk(g_mask_mu);
    if (g_mask_host == nullptr) {
      void* h = nullptr;
      RINGRNN_CUDA_TRY(cudaHostAlloc(&h, sizeof(unsigned long long) * MASK_SLOTS, cudaHostAllocPortable | cudaHostAllocMapped));
      g_mask_host = static_cast<volatile unsigned long long*>(h);
    }
    for (int i = 0; i < MASK_SLOTS && slot < 0; ++i)
      if (!(g_mask_busy & (1u << i))) slot = i;
    if (slot >= 0) g_mask_busy |= 1u << slot;
  }
  if (slot < 0) return RINGRNN_ERR_UNSUPPORTED;  // more than MASK_SLOTS threads asking at once: the caller has another way
  const size_t total = (size_t)rows * a_dim;
  int blocks = (int)((total + 256 * 8 - 1) / (256 * 8));
  blocks = blocks < 1 ? 1 : blocks > 592 ? 592 : blocks;
  cudaError_t e;
  {
    LaunchScope ls(K_PREP, s);
    active_columns_kernel<<<blocks, 256, 0, s>>>(A, (size_t)rows, a_dim, slot, g_mask_host + slot);
    e = cudaGetLastError();
  }
  if (e == cudaSuccess) e = cudaStreamSynchronize(s);
  *mask = g_mask_host[slot];
  {
    std::lock_guard<std::mutex> lk(g_mask_mu);
    g_mask_busy &= ~(1u << slot);
  }
  RINGRNN_CUDA_TRY(e);
  return RINGRNN_OK;
}

extern "C" int ringrnn_decode_angles(long long n, const float* x, const float* y, float* angle, void* stream) {
  if (n <= 0) return RINGRNN_ERR_SHAPE;
  if (!x || !y || !angle) return RINGRNN_ERR_ARG;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  LaunchScope ls(K_LOSS, s);
  decode_angles_kernel<<<grid_for(n), 256, 0, s>>>((size_t)n, aligned16(x, y, angle), x, y, angle);
  RINGRNN_CUDA_TRY(cudaGetLastError());
  return RINGRNN_OK;
}

extern "C" int ringrnn_angular_error(long long n, const float* pred, const float* target, float* error, void* stream) {
  if (n <= 0) return RINGRNN_ERR_SHAPE;
  if (!pred || !target || !error) return RINGRNN_ERR_ARG;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  LaunchScope ls(K_LOSS, s);
  angular_error_kernel<<<grid_for(n), 256, 0, s>>>((size_t)n, aligned16(pred, target, error), pred, target, error);
  RINGRNN_CUDA_TRY(cudaGetLastError());
  return RINGRNN_OK;
}

extern "C" size_t ringrnn_train_bytes(const RingRnnProblem* p) {
  TrainLayout l;
  if (p == nullptr || !train_layout(*p, &l)) return (size_t)-1;
  return l.total;
}

extern "C" int ringrnn_train_step(const RingRnnTrainArgs* a, void* stream) {
  if (a == nullptr) return RINGRNN_ERR_ARG;
  TrainLayout l;
  if (!train_layout(a->p, &l)) return a->p.B <= 0 || a->p.T <= 0 || a->p.N <= 0 ? RINGRNN_ERR_SHAPE : RINGRNN_ERR_UNSUPPORTED;
  if (!a->target || !a->dec_u || !a->dec_v || !a->loss_out) return RINGRNN_ERR_ARG;
  if (a->workspace == nullptr || a->workspace_bytes < l.total || (reinterpret_cast<uintptr_t>(a->workspace) & 255) != 0)
    return RINGRNN_ERR_WORKSPACE;
  char* w = static_cast<char*>(a->workspace);
  const size_t bt = (size_t)a->p.B * a->p.T;
  float* scal = reinterpret_cast<float*>(w + l.scal);
  RingRnnFwdArgs f;
  memset(&f, 0, sizeof(f));
  f.p = a->p;
  f.saved = w + l.saved;
  f.saved_bytes = l.bwd - l.saved;
  f.dec_x = scal; f.dec_y = scal + bt; f.dec_ta = scal + 2 * bt;
  f.dec_u = a->dec_u; f.dec_v = a->dec_v;
  f.final_state = a->final_state;
  f.workspace = w + l.fwd;
  f.workspace_bytes = l.total - l.fwd;
  int rc = ringrnn_fwd(&f, stream);
  if (rc != RINGRNN_OK) return rc;
  rc = ringrnn_angle_loss(a->p.B, a->p.T, f.dec_x, f.dec_y, f.dec_ta, a->target, a->bump_weight, a->inv_count, scal + 3 * bt,
                          scal + 4 * bt, scal + 5 * bt, a->decoded, a->loss_out, reinterpret_cast<float*>(w + l.red), stream);
  if (rc != RINGRNN_OK) return rc;
  RingRnnBwdArgs b;
  memset(&b, 0, sizeof(b));
  b.p = a->p;
  b.coef_x = scal + 3 * bt; b.coef_y = scal + 4 * bt; b.coef_s = scal + 5 * bt;
  b.dec_u = a->dec_u; b.dec_v = a->dec_v;
  b.saved = f.saved; b.saved_bytes = f.saved_bytes;
  b.grad_Wa = a->grad_Wa; b.grad_Wo = a->grad_Wo; b.grad_J = a->grad_J;
  b.workspace = w + l.bwd;
  b.workspace_bytes = l.total - l.bwd;
  return ringrnn_bwd(&b, stream);
}
