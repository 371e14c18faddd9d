// bf16 mode, N <= 512 with up to two active action columns: host side of the kernels of tc_lane.cuh (buffer layouts,
// choice of the samples per unit, weight gradients, checkpoints).
//
// Layouts (NP = 128, 256 or 512, S samples per unit tile, n_ut = ceil(B/S) unit tiles, BPs = n_ut * S):
//   saved            Rh [T+1][NP][BPs] bf16 (slot 0 = r_init, slot t+1 = r_t; the last slot stays unwritten: nothing reads
//                    r_T) | Dh = F'(re), T*NP*BPs bf16 in the threads' own order | sign words, likewise
//   backward scratch DL [T][3][NP][BPs] bf16 = delta, L*delta, R*delta | split-K partials [ns][3*NP][NP] | dJ partials |
//                    dL/dA partial sums [CL][2][T][BPs]
// Neurons are rows and samples are contiguous: what a thread owns (one neuron, S/2 samples) is contiguous, and the weight
// gradient  dW_m[i,j] = sum_t sum_b DL[t][m][i][b] Rh[t][j][b]  is a K-major GEMM, one slab of columns per timestep.
#include <math.h>
#include <stdlib.h>
#include <string.h>

#include "tc_lane.cuh"

namespace ringrnn {

namespace {

struct LaneLayout {
  int NP, CL, S, n_ut, BPs, units;
  size_t rh_slot;  // bytes of one time slot
};

LaneLayout lane_layout(const RingRnnProblem& p) {
  LaneLayout l;
  l.NP = p.N <= 128 ? 128 : p.N <= 256 ? 256 : 512;
  l.CL = l.NP / 128;
  // A step costs its latency chain, which grows with the samples per unit; so the fewest samples at which the batch still
  // fits the 148 SMs in one go.  Beyond 64 per CTA (NP = 128) two units of 64 run side by side in a CTA.
  const int fit = 148 / l.CL;
  l.S = l.NP == 512 || p.B <= 16 * fit ? 16 : p.B <= 32 * fit ? 32 : 64;
  l.n_ut = (p.B + l.S - 1) / l.S;
  l.BPs = l.n_ut * l.S;
  l.units = (l.NP == 128 && l.S == 64 && l.n_ut > fit) ? 2 : 1;
  l.rh_slot = (size_t)l.NP * l.BPs * 2;
  return l;
}

int lane_ckpt_interval(const RingRnnProblem& p) { return (p.ckpt_every > 0 && p.ckpt_every < p.T) ? p.ckpt_every : 0; }
size_t ckpt_slot(const RingRnnProblem& p) { return (size_t)p.B * p.N * sizeof(float); }

size_t sg_bytes(const LaneLayout& l, int T) { return (size_t)T * l.n_ut * l.CL * 2 * (l.S == 64 ? 2 : 1) * 128 * 4; }
size_t every_step_bytes(const LaneLayout& l, int T) {
  return align_up((size_t)(T + 1) * l.rh_slot, 1024) + align_up((size_t)T * l.rh_slot, 1024) + align_up(sg_bytes(l, T), 1024);
}
struct Saved {
  __nv_bfloat16* Rh;
  __nv_bfloat16* Dh;
  uint32_t* Sg;
};
Saved saved_of(void* base, const LaneLayout& l, int T) {
  char* w = static_cast<char*>(base);
  Saved s;
  s.Rh = reinterpret_cast<__nv_bfloat16*>(w);
  w += align_up((size_t)(T + 1) * l.rh_slot, 1024);
  s.Dh = reinterpret_cast<__nv_bfloat16*>(w);
  w += align_up((size_t)T * l.rh_slot, 1024);
  s.Sg = reinterpret_cast<uint32_t*>(w);
  return s;
}

constexpr int FINISH_BLOCKS = 296;

struct LaneBwdLayout {
  size_t dl, partial, jpart, da;
  int nsplit;
};
LaneBwdLayout lane_bwd_layout(const LaneLayout& l, int T) {
  LaneBwdLayout b;
  const int tiles = 3 * l.NP / 128 * (l.NP > 256 ? l.NP / 256 : 1);
  const long long chunks = (long long)T * ((l.BPs + 63) / 64);
  long long ns = 148 / tiles;
  if (ns > chunks / 8) ns = chunks / 8;  // at least eight K chunks per CTA: a partial tile costs as much as a few of them
  b.nsplit = ns < 1 ? 1 : (int)ns;
  b.dl = align_up((size_t)3 * T * l.rh_slot, 1024);
  b.partial = align_up((size_t)b.nsplit * 3 * l.NP * l.NP * 4, 1024);
  b.jpart = align_up(sizeof(double) * 2 * FINISH_BLOCKS, 1024);
  b.da = align_up((size_t)l.CL * 2 * T * l.BPs * 4, 1024);
  return b;
}

// The Wo product and the global inhibition share an accumulator: J1 * (Yo + (J0/J1) * S), see tc_lane.cuh.
template <class P>
void set_inhibition(P& q, float J0, float J1) {
  float ratio = J0;
  q.J1 = 1.f;
  q.use_wo = 0;
  if (J1 != 0.f && fabsf(J0) <= 1e30f * fabsf(J1)) {
    ratio = J0 / J1;
    q.J1 = J1;
    q.use_wo = 1;
  }
  q.n_const = 0;
  for (int i = 0; i < 3; ++i) {  // ratio as a sum of bf16 terms
    const float term = __bfloat162float(__float2bfloat16(ratio));
    q.cterm[i] = term;
    ratio -= term;
    if (term != 0.f) q.n_const = i + 1;
  }
}

// out[k][i] += sum over the parts of add[part][k][i]
__global__ void add_into_kernel(float* o0, float* o1, float* o2, const float* __restrict__ add, int parts, size_t n) {
  float* o = blockIdx.y == 0 ? o0 : blockIdx.y == 1 ? o1 : o2;
  if (o == nullptr) return;
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) {
    float v = o[i];
    for (int p = 0; p < parts; ++p) v += add[((size_t)p * 3 + blockIdx.y) * n + i];
    o[i] = v;
  }
}

// From the split-K partials of dWcat [3*NP][NP]: grad_Wo = J1 * block 0, grad_Wa[colL], [colR] = blocks 1, 2, every other
// column of grad_Wa zero; `add`: on top of what is there (stretches of a checkpointed backward).  With grad_J: dJ0 = sum G,
// dJ1 = sum G*Wo over block 0 in double, block partials in fixed order, the last block to finish adds them up.
__global__ void __launch_bounds__(256) lane_finish_kernel(const float* __restrict__ partial, int nsplit, int N, int NP, float J1,
                                                          int a_dim, int colL, int colR, int add, float* grad_Wo,
                                                          float* grad_Wa, const float* __restrict__ Wo, float* grad_J,
                                                          double* jpart, unsigned* done) {
  __shared__ double s0[8], s1[8];
  __shared__ bool last;
  const size_t NN = (size_t)N * N, slice = (size_t)3 * NP * NP;
  double a0 = 0.0, a1 = 0.0;
  // element (m, i, j) of the three blocks per thread; then the columns of grad_Wa nobody uses
  for (size_t x = blockIdx.x * (size_t)blockDim.x + threadIdx.x; x < 3 * NN; x += (size_t)gridDim.x * blockDim.x) {
    const int m = (int)(x / NN);
    const size_t e = x - m * NN;
    if (m > 0 && (m == 1 ? colL : colR) < 0) continue;
    const int i = (int)(e / N), j = (int)(e - (size_t)i * N);
    const float* src = partial + ((size_t)m * NP + i) * NP + j;
    float v = 0.f;
#pragma unroll 8
    for (int s = 0; s < nsplit; ++s) v += src[s * slice];
    float* o;
    if (m == 0) {
      a0 += v;
      a1 += (double)v * Wo[e];
      v *= J1;
      o = grad_Wo + e;
    } else {
      o = grad_Wa + (size_t)(m == 1 ? colL : colR) * NN + e;
    }
    *o = add ? *o + v : v;
  }
  if (!add && a_dim > (colL >= 0) + (colR >= 0)) {
    const size_t all = (size_t)a_dim * NN;
    for (size_t x = blockIdx.x * (size_t)blockDim.x + threadIdx.x; x < all; x += (size_t)gridDim.x * blockDim.x) {
      const int k = (int)(x / NN);
      if (k != colL && k != colR) grad_Wa[x] = 0.f;
    }
  }
  if (grad_J == nullptr) return;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    a0 += __shfl_down_sync(0xffffffffu, a0, o);
    a1 += __shfl_down_sync(0xffffffffu, a1, o);
  }
  if ((threadIdx.x & 31) == 0) {
    s0[threadIdx.x >> 5] = a0;
    s1[threadIdx.x >> 5] = a1;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int w = 1; w < 8; ++w) {
      s0[0] += s0[w];
      s1[0] += s1[w];
    }
    jpart[2 * blockIdx.x] = s0[0];
    jpart[2 * blockIdx.x + 1] = s1[0];
    __threadfence();
    last = atomicAdd(done, 1u) == gridDim.x - 1;
  }
  __syncthreads();
  if (last && threadIdx.x < 32) {
    __threadfence();
    double x0 = 0.0, x1 = 0.0;
    for (int b = threadIdx.x; b < (int)gridDim.x; b += 32) {
      x0 += jpart[2 * b];
      x1 += jpart[2 * b + 1];
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      x0 += __shfl_down_sync(0xffffffffu, x0, o);
      x1 += __shfl_down_sync(0xffffffffu, x1, o);
    }
    if (threadIdx.x == 0) {
      grad_J[0] = add ? grad_J[0] + (float)x0 : (float)x0;
      grad_J[1] = add ? grad_J[1] + (float)x1 : (float)x1;
      *done = 0u;  // ready for the next stretch
    }
  }
}

// grad_A[b,t0+t,col_k] = sum over the CTAs of part[rank][k][t][b]; other columns are zeroed by the host
__global__ void lane_da_kernel(const float* __restrict__ part, int CL, int B, int T, int BPs, int a_dim, int colL, int colR,
                               float* grad_A, int t0, int T_total) {
  const size_t total = (size_t)B * T;
  for (size_t idx = blockIdx.x * (size_t)blockDim.x + threadIdx.x; idx < total; idx += (size_t)gridDim.x * blockDim.x) {
    const int t = (int)(idx % T), b = (int)(idx / T);
    float* o = grad_A + ((size_t)b * T_total + t0 + t) * a_dim;
    for (int k = 0; k < 2; ++k) {
      const int col = k == 0 ? colL : colR;
      if (col < 0) continue;
      float acc = 0.f;
      for (int r = 0; r < CL; ++r) acc += part[((size_t)(r * 2 + k) * T + t) * BPs + b];
      o[col] = acc;
    }
  }
}

bool aligned16(const void* a) { return (reinterpret_cast<uintptr_t>(a) & 15) == 0; }  // (nullptr is)

// A caller's matrix may be a slice of something larger and start at any float.
void set_weight_loads(LaneFwdParams& q) { q.w_vec = q.N % 4 == 0 && aligned16(q.Wo) && aligned16(q.WL) && aligned16(q.WR); }

template <class P>
void set_common(P& q, const RingRnnProblem& p, const DevProblem& dp, const LaneLayout& l, int T, int t0, int* status, volatile int* host) {
  memset(&q, 0, sizeof(q));
  q.B = p.B; q.T = T; q.N = p.N; q.BPs = l.BPs; q.n_ut = l.n_ut; q.a_dim = p.a_dim;
  q.colL = dp.n_mat > 1 ? dp.cols[0] : -1;
  q.colR = dp.n_mat > 2 ? dp.cols[1] : -1;
  q.alpha = p.alpha;
  set_inhibition(q, p.J0, p.J1);
  const size_t NN = (size_t)p.N * p.N;
  q.Wo = p.Wo;
  q.WL = q.colL >= 0 ? p.Wa + q.colL * NN : nullptr;
  q.WR = q.colR >= 0 ? p.Wa + q.colR * NN : nullptr;
  q.A = p.A;
  q.t0 = t0; q.T_total = p.T;
  q.status = status;
  q.host = host;
}

}  // namespace

// FWD workspace: status(1024) | the other CTAs' decode sums [CL-1][3][B][T]
size_t lane_fwd_workspace_bytes(const RingRnnProblem& p) {
  const LaneLayout l = lane_layout(p);
  return 1024 + (l.CL > 1 ? align_up((size_t)3 * (l.CL - 1) * p.B * p.T * 4, 1024) : 0);
}
size_t lane_saved_bytes(const RingRnnProblem& p) {
  const int K = lane_ckpt_interval(p);
  if (K > 0) return align_up((size_t)((p.T + K - 1) / K) * ckpt_slot(p), 1024);
  return every_step_bytes(lane_layout(p), p.T);
}
size_t lane_bwd_workspace_bytes(const RingRnnProblem& p) {
  const LaneLayout l = lane_layout(p);
  const int K = lane_ckpt_interval(p);
  const LaneBwdLayout b = lane_bwd_layout(l, K > 0 ? K : p.T);
  size_t n = 1024 + b.dl + b.partial + b.jpart + b.da;
  if (K > 0) n += every_step_bytes(l, K) + 2 * align_up(ckpt_slot(p), 1024);
  return n;
}

int lane_forward(const RingRnnFwdArgs& a, const DevProblem& dp, cudaStream_t s) {
  const RingRnnProblem& p = a.p;
  const LaneLayout l = lane_layout(p);
  if (a.workspace == nullptr || a.workspace_bytes < lane_fwd_workspace_bytes(p)) return RINGRNN_ERR_WORKSPACE;
  if ((reinterpret_cast<uintptr_t>(a.workspace) & 255) != 0) return RINGRNN_ERR_WORKSPACE;
  const bool train = a.saved != nullptr;
  if (train && (a.saved_bytes < lane_saved_bytes(p) || (reinterpret_cast<uintptr_t>(a.saved) & 255) != 0))
    return RINGRNN_ERR_WORKSPACE;
  char* w = static_cast<char*>(a.workspace);
  float* dec1 = reinterpret_cast<float*>(w + 1024);
  const int K = train ? lane_ckpt_interval(p) : 0;
  int* status = a.status;
  volatile int* host = nullptr;
  if (status == nullptr) {  // the call's own word, and no copy of it behind the kernels
    status = reinterpret_cast<int*>(w);
    const int rc = host_status_word(&host);
    if (rc != RINGRNN_OK) return rc;
    RINGRNN_CUDA_TRY(cudaMemsetAsync(status, 0, sizeof(int), s));
  }
  if (K > 0)  // checkpoint 0 is the initial state
    RINGRNN_CUDA_TRY(cudaMemcpyAsync(a.saved, p.r_init, ckpt_slot(p), cudaMemcpyDeviceToDevice, s));
  LaneFwdParams q;
  set_common(q, p, dp, l, p.T, 0, status, host);
  set_weight_loads(q);
  q.r_init = p.r_init;
  if (train && K == 0) {
    const Saved sv = saved_of(a.saved, l, p.T);
    q.Rh = sv.Rh; q.Dh = sv.Dh; q.Sg = sv.Sg;
  }
  q.hist = a.bump_history;
  float* const dec[3] = {a.dec_x, a.dec_y, a.dec_ta};
  const bool want_dec = a.dec_x || a.dec_y || a.dec_ta;
  for (int k = 0; k < 3; ++k) {
    q.dec[0][k] = dec[k];
    for (int r = 1; r < l.CL && dec[k] != nullptr; ++r) q.dec[r][k] = dec1 + ((size_t)(r - 1) * 3 + k) * p.B * p.T;
  }
  q.dec_vec = p.T % 4 == 0 && aligned16(a.dec_x) && aligned16(a.dec_y) && aligned16(a.dec_ta) && aligned16(dec1);
  q.dec_u = a.dec_u; q.dec_v = a.dec_v;
  q.final_state = a.final_state;
  q.ckpt = K > 0 ? static_cast<float*>(a.saved) : nullptr;
  q.ckpt_every = K;
  const int rc = lane_forward_launch(p.activation, l.NP, l.S, l.units, q, s);
  if (rc != RINGRNN_OK) return rc;
  if (want_dec && l.CL > 1) {
    LaunchScope ls(K_LOSS, s);
    add_into_kernel<<<dim3(148, 3), 256, 0, s>>>(a.dec_x, a.dec_y, a.dec_ta, dec1, l.CL - 1, (size_t)p.B * p.T);
    RINGRNN_CUDA_TRY(cudaGetLastError());
  }
  return RINGRNN_OK;
}

int lane_backward(const RingRnnBwdArgs& a, const DevProblem& dp, cudaStream_t s) {
  const RingRnnProblem& p = a.p;
  const LaneLayout l = lane_layout(p);
  if (a.workspace == nullptr || a.workspace_bytes < lane_bwd_workspace_bytes(p)) return RINGRNN_ERR_WORKSPACE;
  if ((reinterpret_cast<uintptr_t>(a.workspace) & 255) != 0) return RINGRNN_ERR_WORKSPACE;
  if (a.saved == nullptr || a.saved_bytes < lane_saved_bytes(p) || (reinterpret_cast<uintptr_t>(a.saved) & 255) != 0)
    return RINGRNN_ERR_WORKSPACE;
  const int K = lane_ckpt_interval(p);
  const int Tk = K > 0 ? K : p.T;  // steps of one stretch
  const LaneBwdLayout b = lane_bwd_layout(l, Tk);
  char* w = static_cast<char*>(a.workspace);
  int* status = a.status;
  volatile int* host = nullptr;
  if (status == nullptr) {
    status = reinterpret_cast<int*>(w);
    const int rc = host_status_word(&host);
    if (rc != RINGRNN_OK) return rc;
  }
  unsigned* done = reinterpret_cast<unsigned*>(w + 64);
  if (a.status == nullptr || a.grad_J != nullptr) RINGRNN_CUDA_TRY(cudaMemsetAsync(w, 0, 128, s));  // both words
  w += 1024;
  __nv_bfloat16* DL = reinterpret_cast<__nv_bfloat16*>(w);
  w += b.dl;
  float* partial = reinterpret_cast<float*>(w);
  w += b.partial;
  double* jpart = reinterpret_cast<double*>(w);
  w += b.jpart;
  float* dA_part = reinterpret_cast<float*>(w);
  w += b.da;
  char* chunk_saved = w;
  float* carry[2] = {nullptr, nullptr};
  if (K > 0) {
    w += every_step_bytes(l, K);
    carry[0] = reinterpret_cast<float*>(w);
    carry[1] = reinterpret_cast<float*>(w + align_up(ckpt_slot(p), 1024));
  }
  if (a.grad_A != nullptr && (p.a_dim > 2 || dp.n_mat < 3))
    RINGRNN_CUDA_TRY(cudaMemsetAsync(a.grad_A, 0, sizeof(float) * (size_t)p.B * p.T * p.a_dim, s));

  // With checkpoints the stretches of K steps are taken last to first: each is recomputed from its fp32 state, then run in
  // reverse from the gradient the later stretch handed back, and its weight gradients are added to the total.
  const int n_ck = (p.T + Tk - 1) / Tk;
  for (int c = n_ck - 1; c >= 0; --c) {
    const int t0 = c * Tk, Tc = p.T - t0 < Tk ? p.T - t0 : Tk;
    Saved sv;
    if (K > 0) {
      sv = saved_of(chunk_saved, l, Tc);
      LaneFwdParams f;
      set_common(f, p, dp, l, Tc, t0, status, host);
      set_weight_loads(f);
      f.r_init = static_cast<const float*>(a.saved) + (size_t)c * p.B * p.N;
      f.Rh = sv.Rh; f.Dh = sv.Dh; f.Sg = sv.Sg;
      const int rc = lane_forward_launch(p.activation, l.NP, l.S, l.units, f, s);
      if (rc != RINGRNN_OK) return rc;
    } else {
      sv = saved_of(const_cast<void*>(a.saved), l, p.T);
    }
    LaneBwdParams q;
    set_common(q, p, dp, l, Tc, t0, status, host);
    q.Rh = sv.Rh; q.Dh = sv.Dh; q.Sg = sv.Sg;
    q.grad_output = a.grad_output;
    q.coef_x = a.coef_x; q.coef_y = a.coef_y; q.coef_s = a.coef_s;
    q.dec_u = a.dec_u; q.dec_v = a.dec_v;
    q.DL = DL;
    q.grad_r_init = c == 0 ? a.grad_r_init : carry[c & 1];
    q.dA_part = a.grad_A != nullptr ? dA_part : nullptr;
    q.carry_in = c == n_ck - 1 ? nullptr : carry[(c + 1) & 1];
    int rc = lane_backward_launch(l.NP, l.S, q, s);
    if (rc != RINGRNN_OK) return rc;
    if (a.grad_A != nullptr) {
      LaunchScope ls(K_REDUCE, s);
      lane_da_kernel<<<296, 256, 0, s>>>(dA_part, l.CL, p.B, Tc, l.BPs, p.a_dim, q.colL, q.colR, a.grad_A, t0, p.T);
      RINGRNN_CUDA_TRY(cudaGetLastError());
    }
    const int nsplit = lane_bwd_layout(l, Tc).nsplit;
    rc = tc_gemm_slabs(DL, sv.Rh, partial, 3 * l.NP, l.NP, Tc, l.BPs, nsplit, status, host, s);
    if (rc != RINGRNN_OK) return rc;
    {
      LaunchScope ls(K_REDUCE, s);
      lane_finish_kernel<<<FINISH_BLOCKS, 256, 0, s>>>(partial, nsplit, p.N, l.NP, p.J1, p.a_dim, q.colL, q.colR,
                                                       c == n_ck - 1 ? 0 : 1, a.grad_Wo, a.grad_Wa, p.Wo, a.grad_J, jpart, done);
    }
    RINGRNN_CUDA_TRY(cudaGetLastError());
  }
  return RINGRNN_OK;
}

}  // namespace ringrnn
