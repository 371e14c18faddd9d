// bf16 mode, stepwise variant: one tensor-core GEMM per timestep instead of a persistent kernel.
//
// Used for shapes the persistent tcgen05 kernels do not take, or would leave most of the machine idle on (training_route in
// ringrnn_bf16.cu has the lines).  Replaces, for those shapes, the same reference kernels as the persistent path
// (cpp/kernels/fwd_1loop_tc_idx.cuh:265-277 and the five per-step launches of
// cpp/kernels/bwd_mixed_precision_aggressive.cuh:564-671), without materialising W_eff[B,N,N].
//
// With m = 0 for Wo and m = 1..n for the active action matrices (coefficient c_0 = 1 -- J1 is folded into the
// stacked weights -- and c_m = A[b,t,cols[m-1]]), both directions form all products of a step with one GEMM and mix them
// in fp32 in the row kernel:
//   forward   Z_t = r_{t-1} . Wf^T,  Wf[m*NP + i, j] = W_m[i,j]     ([BP,NP] x [NP,(1+n)NP] per step)
//             re_t[b,i] = J0 sum_j r_{t-1}[b,j] + sum_m c_m Z_t[b, m*NP + i]
//   backward  Z_t = delta_t . Wt^T,  Wt[m*NP + j, i] = W_m[i,j]
//             carry[b,j] = (1-alpha) g_t[b,j] + J0 sum_i delta_t[b,i] + sum_m c_m Z_t[b, m*NP + j]
//             dL/dA[b,t,cols[k]] = sum_j r_{t-1}[b,j] Z_t[b,(1+k)*NP + j]
//   weights   dWst = sum_t delta_t^T X_t, X_t[b, m*NP + j] = c_m r_{t-1}[b,j]: one split-K GEMM over all (t, b) at the end.
// Between the GEMMs a row kernel (one block per sample) applies the epilogue of one step and prepares the operand
// of the next, so a step costs two launches.  Split-K partial sums are reduced in fixed order: bit-reproducible.
//
// Forward, large batches (the [BP,NP] output alone fills the machine): re_t = X_t . Wst^T with the scaled copies of the state
// as one long operand, because Z would be (1+n) times the output.
#include <string.h>

#include "ringrnn_common.cuh"
#include "tc_ptx.cuh"

namespace ringrnn {

namespace {

constexpr int ROW_MAX = 512;  // threads of a row kernel: four neurons each, several rounds beyond 2048

struct SwCols {
  int n;
  int c[RINGRNN_MAX_ACTIVE];
};

struct SwLayout {
  int NP, BP, n_act, blocks;  // blocks = 1 + n_act column blocks of NP
  long long KX;               // (1 + n_act) * NP
  bool concat;                // forward: one long operand X instead of all products Z
  int nt_z, ns_z;             // tile width and split-K factor of the Z GEMM
};

int sw_active(const RingRnnProblem& p) { return p.n_active < 0 ? p.a_dim : p.n_active; }

int splits_for(long long tiles, long long K) {
  long long ns = 148 / (tiles > 0 ? tiles : 1);
  while (ns > 1 && K / ns < 512) --ns;
  return (int)(ns < 1 ? 1 : ns);
}

// Tile width and K splits of the Z GEMM by estimated cycles: waves of 148 CTAs x (start-up + operand bytes at the 50 B/clk
// that enter an SM + the tile's way out at about 24 B/clk), plus the partial sums written and read back at 2.5 KB/clk.
// CTA pairs (an even number of row tiles) fetch half of the B rows each.
void z_shape(int BP, long long KX, int K, int* nt_out, int* ns_out) {
  const bool pair = BP % 256 == 0;
  double best = 1e300;
  for (int nt = 512; nt >= 128; nt /= 2) {
    if (KX % nt != 0) continue;
    for (int ns = 1; ns <= 8 && K / ns >= 128; ++ns) {
      const double ctas = (double)(BP / 128) * (KX / nt) * ns;
      const long long chunks = (K / 64 + ns - 1) / ns;
      const double waves = (double)(((long long)ctas + 147) / 148);
      const double cost = waves * (1500 + chunks * (128.0 + (pair ? nt / 2 : nt)) * 128 / 50 + nt * 512.0 / 24) + 8.0 * ns * BP * KX / 2500;
      if (cost < best) {
        best = cost;
        *nt_out = nt;
        *ns_out = ns;
      }
    }
  }
}

SwLayout sw_layout(const RingRnnProblem& p) {
  SwLayout l;
  l.NP = (p.N + 127) / 128 * 128;
  l.BP = (p.B + 127) / 128 * 128;
  l.n_act = sw_active(p);
  l.blocks = 1 + l.n_act;
  l.KX = (long long)l.blocks * l.NP;
  const int nt_fwd = (l.NP % 512 == 0) ? 512 : (l.NP % 256 == 0) ? 256 : 128;
  l.concat = splits_for((long long)(l.BP / 128) * (l.NP / nt_fwd), l.KX) == 1;
  z_shape(l.BP, l.KX, l.NP, &l.nt_z, &l.ns_z);
  return l;
}
// split-K factor of the weight-gradient GEMM over T steps
int dw_splits(const SwLayout& l, int T) {
  const int nt_dw = (l.KX % 512 == 0) ? 512 : (l.KX % 256 == 0) ? 256 : 128;
  return splits_for((long long)(l.NP / 128) * (l.KX / nt_dw), (long long)T * l.BP);
}
int sw_ckpt_interval(const RingRnnProblem& p) { return (p.ckpt_every > 0 && p.ckpt_every < p.T) ? p.ckpt_every : 0; }
size_t ckpt_slot(const RingRnnProblem& p) { return sizeof(float) * (size_t)p.B * p.N; }

int row_threads(int NP) { return NP / 4 < ROW_MAX ? NP / 4 : ROW_MAX; }  // NP is a multiple of 128

// four consecutive elements
__device__ __forceinline__ float4 ld4(const float* p) { return *reinterpret_cast<const float4*>(p); }
__device__ __forceinline__ void st4(float* p, float4 v) { *reinterpret_cast<float4*>(p) = v; }
__device__ __forceinline__ uint2 to_bf16x4(float4 v) {
  const __nv_bfloat162 a = __floats2bfloat162_rn(v.x, v.y), b = __floats2bfloat162_rn(v.z, v.w);
  return make_uint2(*reinterpret_cast<const uint32_t*>(&a), *reinterpret_cast<const uint32_t*>(&b));
}
__device__ __forceinline__ float4 of_bf16x4(uint2 v) {
  return make_float4(__uint_as_float(v.x << 16), __uint_as_float(v.x & 0xffff0000u), __uint_as_float(v.y << 16),
                     __uint_as_float(v.y & 0xffff0000u));
}
// elements i .. i+3 of a caller's row of N: single floats where the row ends or starts off a 16-byte boundary
__device__ __forceinline__ float4 row_ld(const float* row, int i, int N, bool vec) {
  if (vec && i + 3 < N) return __ldg(reinterpret_cast<const float4*>(row + i));
  return make_float4(i < N ? __ldg(row + i) : 0.f, i + 1 < N ? __ldg(row + i + 1) : 0.f, i + 2 < N ? __ldg(row + i + 2) : 0.f,
                     i + 3 < N ? __ldg(row + i + 3) : 0.f);
}
__device__ __forceinline__ void row_st(float* row, int i, int N, bool vec, float4 v) {
  if (vec && i + 3 < N) {
    st4(row + i, v);
  } else {
    if (i < N) row[i] = v.x;
    if (i + 1 < N) row[i + 1] = v.y;
    if (i + 2 < N) row[i + 2] = v.z;
    if (i + 3 < N) row[i + 3] = v.w;
  }
}
__device__ __forceinline__ float4 fma4(float c, float4 x, float4 y) {
  return make_float4(fmaf(c, x.x, y.x), fmaf(c, x.y, y.y), fmaf(c, x.z, y.z), fmaf(c, x.w, y.w));
}
__device__ __forceinline__ float sum4(float4 v) { return (v.x + v.y) + (v.z + v.w); }
__device__ __forceinline__ float dot4(float4 a, float4 b) { return fmaf(a.x, b.x, a.y * b.y) + fmaf(a.z, b.z, a.w * b.w); }

// block-wide sum; every thread gets the result
__device__ __forceinline__ float block_sum(float v, float* red) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  __syncthreads();  // red may still be read from the previous call
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = v;
  __syncthreads();
  float tot = 0.f;
  for (int w = 0; w < (int)(blockDim.x >> 5); ++w) tot += red[w];
  return tot;
}

// bf16 copy of the matrices, zero padded, block 0 scaled by J1: element (i, j) of block m at i*ld_i + m*ld_m + j.
// grid (x, blocks), block 256.  Bound by memory: 4 bytes in and 2 out per element, 17 matrices of 2048^2 (428 MB) in 67 us =
// 6.4 TB/s.
__global__ void __launch_bounds__(256) sw_prep_weights_kernel(const float* __restrict__ Wo, const float* __restrict__ Wa,
                                                              SwCols cols, float J1, int N, int NP, long long ld_i,
                                                              long long ld_m, bool vec, __nv_bfloat16* __restrict__ out) {
  const int m = blockIdx.y;
  const float* W = (m == 0) ? Wo : Wa + (size_t)cols.c[m - 1] * N * N;
  const float scale = (m == 0) ? J1 : 1.f;
  const int quads = NP / 4, total = NP * quads, stride = gridDim.x * 256;
#pragma unroll 4
  for (int e = blockIdx.x * 256 + threadIdx.x; e < total; e += stride) {
    const int i = e / quads, j = (e - i * quads) * 4;
    float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
    if (i < N) v = row_ld(W + (size_t)i * N, j, N, vec);
    v.x *= scale; v.y *= scale; v.z *= scale; v.w *= scale;
    *reinterpret_cast<uint2*>(out + i * ld_i + m * ld_m + j) = to_bf16x4(v);
  }
}

// The transposed copy for reverse time, out[m*NP + j][i] = W_m[i][j], by tiles of 32 x 32.  grid (NP/32, NP/32, blocks), block 256
__global__ void __launch_bounds__(256) sw_prep_transposed_kernel(const float* __restrict__ Wo, const float* __restrict__ Wa,
                                                                 SwCols cols, float J1, int N, int NP,
                                                                 __nv_bfloat16* __restrict__ out) {
  __shared__ float tile[32][33];
  const int m = blockIdx.z, j0 = blockIdx.x * 32, i0 = blockIdx.y * 32;
  const float* W = (m == 0) ? Wo : Wa + (size_t)cols.c[m - 1] * N * N;
  const float scale = (m == 0) ? J1 : 1.f;
  const int c = threadIdx.x & 31;
#pragma unroll
  for (int r = threadIdx.x >> 5; r < 32; r += 8)
    tile[r][c] = (i0 + r < N && j0 + c < N) ? scale * __ldg(W + (size_t)(i0 + r) * N + j0 + c) : 0.f;
  __syncthreads();
  const int j = threadIdx.x >> 3, i = (threadIdx.x & 7) * 4;
  *reinterpret_cast<uint2*>(out + ((size_t)m * NP + j0 + j) * NP + i0 + i) =
      to_bf16x4(make_float4(tile[i][j], tile[i + 1][j], tile[i + 2][j], tile[i + 3][j]));
}

// A pass may cover steps [t0, t0 + T) of a sequence of T_total (a stretch between checkpoints): the action signal, the decode
// sums, grad_output and the loss coefficients are indexed with the global step, everything else with the local one.
struct SwFwd {
  int B, T, N, NP, BP, a_dim, nsplit, t0, T_total;
  long long KX;
  bool concat;             // partial [nsplit = 1][BP][NP] and X; otherwise Z [nsplit][BP][KX]
  bool vec;                // the caller's rows of N floats start on 16-byte boundaries
  float J0, alpha;
  const float* A;
  const float* r_init;
  const float* partial;
  float* state;            // [BP][NP] fp32 master state
  float* rowsum;           // [BP]
  __nv_bfloat16* X;        // [BP][KX] (concat) or [BP][NP] or nullptr: the operand of the next step, unless Rh is it
  __nv_bfloat16* Rh;       // [T+1][BP][NP] or nullptr
  __nv_bfloat16* Dh;       // [T][BP][NP] or nullptr
  float* hist;             // [T,B,N] or nullptr
  float* final_state;      // [B,N] or nullptr
  float* dec_x;            // [B,T] or nullptr
  float* dec_y;
  float* dec_ta;
  const float* dec_u;
  const float* dec_v;
  float* ckpt;             // [ceil(T/ckpt_every)][B][N]: slot c receives the state after step c*ckpt_every - 1, or nullptr
  int ckpt_every;
  SwCols cols;
};

// One block per padded sample row, four neurons per thread.  t >= 0: finishes step t (r_t from the GEMM of step t), then
// builds the operand of step t+1.  t = -1: loads r_init and builds the operand of step 0.  Bound by the latency of its
// loads: all of a thread's products of a step are in flight together (one float at a time, eight neurons per thread in turn:
// 256 samples of N = 2048 with 18 partial sums took about 40 us, now 12 with the products coming from HBM).
template <int ACT>
__global__ void __launch_bounds__(ROW_MAX) sw_forward_row_kernel(SwFwd q, int t) {
  __shared__ float red[ROW_MAX / 32];
  __shared__ float coef[1 + RINGRNN_MAX_ACTIVE];  // of step t (products) or, concat, of step t+1 (operand)
  const int b = blockIdx.x, n = q.cols.n;
  const bool valid = b < q.B;
  float* st = q.state + (size_t)b * q.NP;
  float px = 0.f, py = 0.f, pa = 0.f, rs = 0.f;
  const bool build = t + 1 < q.T;
  const int t_c = q.concat ? t + 1 : t;
  for (int k = threadIdx.x; k <= n; k += blockDim.x)
    coef[k] = k == 0 ? 1.f : (valid && t_c >= 0 && t_c < q.T) ? __ldg(q.A + ((size_t)b * q.T_total + q.t0 + t_c) * q.a_dim + q.cols.c[k - 1]) : 0.f;
  const float s_prev = (t >= 0) ? q.rowsum[b] : 0.f;
  __syncthreads();
  const int blocks = q.concat ? 1 : 1 + n;
  const size_t ld = q.concat ? q.NP : q.KX;
  const bool dec = q.dec_x != nullptr || q.dec_y != nullptr;
  for (int i = threadIdx.x * 4; i < q.NP; i += blockDim.x * 4) {
    float r[4] = {0.f, 0.f, 0.f, 0.f};
    if (t < 0) {
      if (valid) {
        const float4 r0 = row_ld(q.r_init + (size_t)b * q.N, i, q.N, q.vec);
        r[0] = r0.x; r[1] = r0.y; r[2] = r0.z; r[3] = r0.w;
      }
    } else {
      float d[4] = {0.f, 0.f, 0.f, 0.f};
      if (valid) {
        float4 z = make_float4(0.f, 0.f, 0.f, 0.f);
        for (int s = 0; s < q.nsplit; ++s) {
          const float* src = q.partial + ((size_t)s * q.BP + b) * ld + i;
#pragma unroll 8
          for (int m = 0; m < blocks; ++m) z = fma4(coef[m], ld4(src + (size_t)m * q.NP), z);
        }
        const float zz[4] = {z.x, z.y, z.z, z.w};
        const float4 old4 = ld4(st + i);
        const float old[4] = {old4.x, old4.y, old4.z, old4.w};
#pragma unroll
        for (int x = 0; x < 4; ++x)
          if (i + x < q.N) {
            const float re = fmaf(q.J0, s_prev, zz[x]);
            r[x] = fmaf(q.alpha, act_fn<ACT>(re), (1.f - q.alpha) * old[x]);
            if (q.Dh != nullptr) d[x] = act_grad<ACT>(re);
            if (dec) {
              px = fmaf(r[x], q.dec_u[i + x], px);
              py = fmaf(r[x], q.dec_v[i + x], py);
            }
            pa += fabsf(r[x]);
          }
        const float4 r4 = make_float4(r[0], r[1], r[2], r[3]);
        if (q.hist != nullptr) row_st(q.hist + ((size_t)t * q.B + b) * q.N, i, q.N, q.vec, r4);
        if (q.ckpt != nullptr && t + 1 < q.T && (t + 1) % q.ckpt_every == 0)
          row_st(q.ckpt + ((size_t)((t + 1) / q.ckpt_every) * q.B + b) * q.N, i, q.N, q.vec, r4);
        if (q.final_state != nullptr && t + 1 == q.T) row_st(q.final_state + (size_t)b * q.N, i, q.N, q.vec, r4);
      }
      if (q.Dh != nullptr)
        *reinterpret_cast<uint2*>(q.Dh + ((size_t)t * q.BP + b) * q.NP + i) = to_bf16x4(make_float4(d[0], d[1], d[2], d[3]));
    }
    st4(st + i, make_float4(r[0], r[1], r[2], r[3]));
    const uint2 rb = to_bf16x4(make_float4(r[0], r[1], r[2], r[3]));
    const float4 rf = of_bf16x4(rb);
    rs += sum4(rf);
    if (q.Rh != nullptr) *reinterpret_cast<uint2*>(q.Rh + ((size_t)(t + 1) * q.BP + b) * q.NP + i) = rb;
    if (build && q.X != nullptr) {
      __nv_bfloat16* x = q.X + (size_t)b * (q.concat ? q.KX : (long long)q.NP) + i;
      *reinterpret_cast<uint2*>(x) = rb;
      if (q.concat)
        for (int k = 1; k <= n; ++k) {
          const float c = coef[k];
          *reinterpret_cast<uint2*>(x + (size_t)k * q.NP) = to_bf16x4(make_float4(c * rf.x, c * rf.y, c * rf.z, c * rf.w));
        }
    }
  }
  if (build) {
    const float tot = block_sum(rs, red);
    if (threadIdx.x == 0) q.rowsum[b] = tot;
  }
  if (t >= 0 && valid && (dec || q.dec_ta != nullptr)) {
    const float sx = block_sum(px, red), sy = block_sum(py, red), sa = block_sum(pa, red);
    if (threadIdx.x == 0) {
      const size_t o = (size_t)b * q.T_total + q.t0 + t;
      if (q.dec_x != nullptr) q.dec_x[o] = sx;
      if (q.dec_y != nullptr) q.dec_y[o] = sy;
      if (q.dec_ta != nullptr) q.dec_ta[o] = sa;
    }
  }
}

struct SwBwd {
  int B, T, N, NP, BP, a_dim, nsplit, t0, T_total;
  bool resume;               // the first carry is what the stretch after this one left in g; otherwise zero
  long long KX;
  bool vec;                  // as in SwFwd
  float J0, alpha;
  const float* A;
  const float* grad_output;  // [T,B,N] or nullptr
  const float* coef_x;       // [B,T] or nullptr
  const float* coef_y;
  const float* coef_s;
  const float* dec_u;
  const float* dec_v;
  const __nv_bfloat16* Rh;   // [T+1][BP][NP]
  const __nv_bfloat16* Dh;   // [T][BP][NP]
  const float* partial;      // [nsplit][BP][KX]: Z of the step whose carry is formed
  float* g;                  // [BP][NP] fp32: g_t of the step in flight
  float* sum_delta;          // [BP]
  __nv_bfloat16* Delta;      // [T][BP][NP]
  float* grad_r_init;        // [B,N] or nullptr
  float* grad_A;             // [B,T,a_dim] or nullptr (pre-zeroed)
  SwCols cols;
};

// One block per padded sample row, four neurons per thread.  t_carry >= 0: forms the carry out of step t_carry from Z (and
// dL/dA of that step, WANT_DA); t_delta >= 0: g and delta of step t_delta from the carry (zero when t_carry < 0).
template <bool WANT_DA>
__global__ void __launch_bounds__(ROW_MAX) sw_backward_row_kernel(SwBwd q, int t_carry, int t_delta) {
  __shared__ float red[ROW_MAX / 32];
  __shared__ float coef[1 + RINGRNN_MAX_ACTIVE];
  __shared__ float da[WANT_DA ? (1 + RINGRNN_MAX_ACTIVE) * (ROW_MAX / 32) : 1];  // [matrix][warp]
  const int b = blockIdx.x, n = q.cols.n, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const bool valid = b < q.B;
  float* g = q.g + (size_t)b * q.NP;
  const float beta = 1.f - q.alpha;
  float cx = 0.f, cy = 0.f, cs = 0.f;
  if (valid && t_delta >= 0 && q.coef_x != nullptr) {
    const size_t bt = (size_t)b * q.T_total + q.t0 + t_delta;
    cx = q.coef_x[bt];
    cy = q.coef_y[bt];
    cs = q.coef_s[bt];
  }
  for (int k = threadIdx.x; k <= n; k += blockDim.x)
    coef[k] = k == 0 ? 1.f : (valid && t_carry >= 0) ? __ldg(q.A + ((size_t)b * q.T_total + q.t0 + t_carry) * q.a_dim + q.cols.c[k - 1]) : 0.f;
  if (WANT_DA)
    for (int x = threadIdx.x; x < (1 + n) * (ROW_MAX / 32); x += blockDim.x) da[x] = 0.f;
  const float sd = (t_carry >= 0) ? q.sum_delta[b] : 0.f;
  __syncthreads();
  float ds = 0.f;
  for (int j = threadIdx.x * 4; j < q.NP; j += blockDim.x * 4) {  // whole warps: NP is a multiple of 128
    float4 carry = make_float4(0.f, 0.f, 0.f, 0.f);
    if (t_carry >= 0 && valid) {
      float4 rp = make_float4(0.f, 0.f, 0.f, 0.f);  // (zero beyond N)
      if (WANT_DA) rp = of_bf16x4(*reinterpret_cast<const uint2*>(q.Rh + ((size_t)t_carry * q.BP + b) * q.NP + j));
      for (int s = 0; s < q.nsplit; ++s) {
        const float* src = q.partial + ((size_t)s * q.BP + b) * q.KX + j;
#pragma unroll 8
        for (int m = 0; m <= n; ++m) {
          const float4 z = ld4(src + (size_t)m * q.NP);
          carry = fma4(coef[m], z, carry);
          if (WANT_DA && m > 0) {
            float v = dot4(rp, z);
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
            if (lane == 0) da[m * (ROW_MAX / 32) + warp] += v;
          }
        }
      }
      const float4 go = ld4(g + j);
      const float js = q.J0 * sd;
      carry = make_float4(carry.x + fmaf(beta, go.x, js), carry.y + fmaf(beta, go.y, js), carry.z + fmaf(beta, go.z, js),
                          carry.w + fmaf(beta, go.w, js));
    } else if (t_carry < 0 && q.resume) {
      carry = ld4(g + j);
    }
    if (t_delta >= 0) {
      float gg[4] = {carry.x, carry.y, carry.z, carry.w};
      float4 go = make_float4(0.f, 0.f, 0.f, 0.f), rt = go;
      if (valid && q.grad_output != nullptr) go = row_ld(q.grad_output + ((size_t)(q.t0 + t_delta) * q.B + b) * q.N, j, q.N, q.vec);
      if (valid && q.coef_x != nullptr)
        rt = of_bf16x4(*reinterpret_cast<const uint2*>(q.Rh + ((size_t)(t_delta + 1) * q.BP + b) * q.NP + j));
      const float gs[4] = {go.x, go.y, go.z, go.w}, rr[4] = {rt.x, rt.y, rt.z, rt.w};
      const float4 dact = of_bf16x4(*reinterpret_cast<const uint2*>(q.Dh + ((size_t)t_delta * q.BP + b) * q.NP + j));
#pragma unroll
      for (int x = 0; x < 4; ++x) {
        if (!valid || j + x >= q.N) {
          gg[x] = 0.f;
          continue;
        }
        gg[x] += gs[x];
        if (q.coef_x != nullptr) {
          gg[x] = fmaf(cx, q.dec_u[j + x], gg[x]);
          gg[x] = fmaf(cy, q.dec_v[j + x], gg[x]);
          gg[x] = fmaf(cs, (rr[x] > 0.f) ? 1.f : ((rr[x] < 0.f) ? -1.f : 0.f), gg[x]);
        }
      }
      st4(g + j, make_float4(gg[0], gg[1], gg[2], gg[3]));
      const uint2 db = to_bf16x4(make_float4(q.alpha * dact.x * gg[0], q.alpha * dact.y * gg[1], q.alpha * dact.z * gg[2],
                                             q.alpha * dact.w * gg[3]));
      *reinterpret_cast<uint2*>(q.Delta + ((size_t)t_delta * q.BP + b) * q.NP + j) = db;
      ds += sum4(of_bf16x4(db));
    } else {
      if (valid && q.grad_r_init != nullptr) row_st(q.grad_r_init + (size_t)b * q.N, j, q.N, q.vec, carry);
      if (q.t0 > 0) st4(g + j, carry);
    }
  }
  if (t_delta >= 0) {
    const float tot = block_sum(ds, red);
    if (threadIdx.x == 0) q.sum_delta[b] = tot;
  }
  if (WANT_DA && t_carry >= 0 && valid) {
    __syncthreads();
    for (int k = threadIdx.x; k < n; k += blockDim.x) {
      float v = 0.f;
      for (int w = 0; w < (int)(blockDim.x >> 5); ++w) v += da[(1 + k) * (ROW_MAX / 32) + w];
      q.grad_A[((size_t)b * q.T_total + q.t0 + t_carry) * q.a_dim + q.cols.c[k]] = v;
    }
  }
}

// Xall[t][b][m*NP + j] = c_m(b,t) * r_{t-1}[b,j] for all t: the B operand of the weight-gradient GEMM.
// grid (BP, T or as many rows as a grid may have), four neurons per thread
constexpr int MAX_GRID_Y = 65535;
__global__ void __launch_bounds__(ROW_MAX) sw_build_xall_kernel(const __nv_bfloat16* __restrict__ Rh, const float* __restrict__ A,
                                                                SwCols cols, int B, int T, int t0, int T_total, int a_dim, int NP,
                                                                int BP, long long KX, __nv_bfloat16* __restrict__ Xall) {
  const int b = blockIdx.x;
  const bool valid = b < B;
  for (int t = blockIdx.y; t < T; t += gridDim.y) {
    const __nv_bfloat16* r = Rh + ((size_t)t * BP + b) * NP;
    __nv_bfloat16* x = Xall + ((size_t)t * BP + b) * KX;
    const float* at = A + ((size_t)b * T_total + t0 + t) * a_dim;
    for (int j = threadIdx.x * 4; j < NP; j += blockDim.x * 4) {
      const uint2 rb = *reinterpret_cast<const uint2*>(r + j);
      const float4 rf = of_bf16x4(rb);
      *reinterpret_cast<uint2*>(x + j) = rb;
#pragma unroll 4
      for (int k = 0; k < cols.n; ++k) {
        const float c = valid ? __ldg(at + cols.c[k]) : 0.f;
        *reinterpret_cast<uint2*>(x + (size_t)(1 + k) * NP + j) = to_bf16x4(make_float4(c * rf.x, c * rf.y, c * rf.z, c * rf.w));
      }
    }
  }
}

__global__ void sw_accumulate_kernel(float* __restrict__ out, const float* __restrict__ in, size_t n) {
  for (size_t e = blockIdx.x * (size_t)blockDim.x + threadIdx.x; e < n; e += (size_t)gridDim.x * blockDim.x) out[e] += in[e];
}

// dWst [NP][KX] -> grad_Wo = J1 * block 0 (the operand block 0 is the unscaled state), raw = block 0,
// grad_Wa[cols[k]] = block 1 + k
__global__ void sw_unpack_dw_kernel(const float* __restrict__ dWst, int N, int NP, long long KX, float J1, SwCols cols,
                                    float* grad_Wo, float* grad_Wa, float* raw) {
  const size_t NN = (size_t)N * N;
  for (size_t e = blockIdx.x * (size_t)blockDim.x + threadIdx.x; e < NN; e += (size_t)gridDim.x * blockDim.x) {
    const int i = (int)(e / N), j = (int)(e % N);
    const float g0 = dWst[(size_t)i * KX + j];
    grad_Wo[e] = J1 * g0;
    raw[e] = g0;
    for (int k = 0; k < cols.n; ++k) grad_Wa[(size_t)cols.c[k] * NN + e] = dWst[(size_t)i * KX + (size_t)(1 + k) * NP + j];
  }
}

SwCols cols_of(const DevProblem& dp) {
  SwCols c;
  c.n = dp.n_mat - 1;
  for (int k = 0; k < c.n; ++k) c.c[k] = dp.cols[k];
  return c;
}

template <class K, class... Args>
cudaError_t launch_row(K kernel, int rows, int NP, cudaStream_t s, Args... args) {
  kernel<<<rows, row_threads(NP), 0, s>>>(args...);
  return cudaGetLastError();
}

template <int ACT>
void launch_forward_row(const SwFwd& q, int t, cudaStream_t s) {
  LaunchScope ls(K_FWD, s);
  launch_row(sw_forward_row_kernel<ACT>, q.BP, q.NP, s, q, t);
}

void forward_row(int act, const SwFwd& q, int t, cudaStream_t s) {
  switch (act) {
    case RINGRNN_ACT_RELU: launch_forward_row<RINGRNN_ACT_RELU>(q, t, s); break;
    case RINGRNN_ACT_GELU: launch_forward_row<RINGRNN_ACT_GELU>(q, t, s); break;
    case RINGRNN_ACT_SILU: launch_forward_row<RINGRNN_ACT_SILU>(q, t, s); break;
    default: launch_forward_row<RINGRNN_ACT_TANH>(q, t, s); break;
  }
}

}  // namespace

// Any N (padded to a multiple of 128) and up to RINGRNN_MAX_ACTIVE active columns; the stacked operand of one step
// must stay below 2^31 elements per row block for the GEMM's 32-bit extents.
bool stepwise_supported(const RingRnnProblem& p) {
  const int n_act = sw_active(p);
  if (p.B < 1 || p.T < 1 || p.N < 1 || n_act > RINGRNN_MAX_ACTIVE) return false;
  const long long NP = (p.N + 127) / 128 * 128;
  return NP <= 16384 && (1 + n_act) * NP <= (1ll << 30);
}

namespace {
size_t x_bytes(const SwLayout& l) { return align_up((size_t)l.BP * (l.concat ? l.KX : l.NP) * 2, 1024); }
size_t z_bytes(const SwLayout& l, bool concat) {
  return align_up((concat ? (size_t)l.BP * l.NP : (size_t)l.ns_z * l.BP * l.KX) * 4, 1024);
}
bool aligned16(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15) == 0; }  // (nullptr is)
int prep_blocks(const SwLayout& l) {
  const long long n = (long long)l.NP * l.NP / 4 / (256 * 4);
  return n < 1 ? 1 : n > 592 ? 592 : (int)n;
}
}  // namespace

// FWD workspace: status(1024) | weights | X | state | rowsum | products
size_t stepwise_fwd_workspace_bytes(const RingRnnProblem& p) {
  const SwLayout l = sw_layout(p);
  return 1024 + align_up((size_t)l.NP * l.KX * 2, 1024) + x_bytes(l) + align_up((size_t)l.BP * l.NP * 4, 1024) +
         align_up((size_t)l.BP * 4, 1024) + z_bytes(l, l.concat);
}
// SAVED: Rh [T+1][BP][NP] | Dh [T][BP][NP] (bf16); with checkpoints fp32 states [ceil(T/K)][B][N]
static size_t every_step_bytes(const SwLayout& l, int T) {
  return align_up((size_t)(T + 1) * l.BP * l.NP * 2, 1024) + align_up((size_t)T * l.BP * l.NP * 2, 1024);
}
size_t stepwise_saved_bytes(const RingRnnProblem& p) {
  const int K = sw_ckpt_interval(p);
  if (K > 0) return align_up((size_t)((p.T + K - 1) / K) * ckpt_slot(p), 1024);
  return every_step_bytes(sw_layout(p), p.T);
}
// BWD workspace (K = p.T without checkpoints): status(1024) | WstT | Delta [K][BP][NP] | g | sum_delta | Z | Xall [K][BP][KX] |
//                dW partials | dWst | raw; with checkpoints also weights | X | state | rowsum | saved stretch | dWst of a stretch
size_t stepwise_bwd_workspace_bytes(const RingRnnProblem& p) {
  const SwLayout l = sw_layout(p);
  const int K = sw_ckpt_interval(p), T = K > 0 ? K : p.T;
  const size_t w_bytes = align_up((size_t)l.KX * l.NP * 2, 1024), dw_bytes = align_up((size_t)l.NP * l.KX * 4, 1024);
  const size_t state_bytes = align_up((size_t)l.BP * l.NP * 4, 1024), row_bytes = align_up((size_t)l.BP * 4, 1024);
  size_t n = 1024 + w_bytes + align_up((size_t)T * l.BP * l.NP * 2, 1024) + state_bytes + row_bytes + z_bytes(l, false) +
             align_up((size_t)T * l.BP * l.KX * 2, 1024) + align_up((size_t)dw_splits(l, T) * l.NP * l.KX * 4, 1024) + dw_bytes +
             align_up((size_t)p.N * p.N * 4, 1024);
  if (K > 0) n += w_bytes + x_bytes(l) + state_bytes + row_bytes + every_step_bytes(l, K) + dw_bytes;
  return n;
}

namespace {

struct SwFwdBuffers {
  __nv_bfloat16* W;
  __nv_bfloat16* X;
  float* state;
  float* rowsum;
  float* partial;
  int* status;
};

int prepare_forward(const RingRnnProblem& p, const DevProblem& dp, const SwLayout& l, const SwFwdBuffers& m, cudaStream_t s) {
  LaunchScope ls(K_PREP, s);
  const bool vec = p.N % 4 == 0 && aligned16(p.Wo) && aligned16(dp.Wa);
  sw_prep_weights_kernel<<<dim3(prep_blocks(l), l.blocks), 256, 0, s>>>(p.Wo, dp.Wa, cols_of(dp), p.J1, p.N, l.NP,
                                                                        l.concat ? l.KX : l.NP,
                                                                        l.concat ? l.NP : (long long)l.NP * l.NP, vec, m.W);
  RINGRNN_CUDA_TRY(cudaGetLastError());
  return RINGRNN_OK;
}

// Steps [q.t0, q.t0 + q.T) from q.r_init; the caller has set the outputs it wants.
int run_forward(const RingRnnProblem& p, const DevProblem& dp, const SwLayout& l, const SwFwdBuffers& m, SwFwd q, cudaStream_t s) {
  q.B = p.B; q.N = p.N; q.NP = l.NP; q.BP = l.BP; q.a_dim = p.a_dim; q.nsplit = l.concat ? 1 : l.ns_z;
  q.T_total = p.T;
  q.concat = l.concat;
  q.vec = p.N % 4 == 0 && aligned16(q.r_init) && aligned16(q.hist) && aligned16(q.final_state) && aligned16(q.ckpt);
  q.KX = l.KX; q.J0 = p.J0; q.alpha = p.alpha;
  q.A = p.A; q.partial = m.partial; q.state = m.state; q.rowsum = m.rowsum;
  q.X = l.concat || q.Rh == nullptr ? m.X : nullptr;
  q.cols = cols_of(dp);
  forward_row(p.activation, q, -1, s);
  RINGRNN_CUDA_TRY(cudaGetLastError());
  for (int t = 0; t < q.T; ++t) {
    int rc;
    if (l.concat)
      rc = tc_gemm(0, m.X, m.W, m.partial, nullptr, l.BP, l.NP, l.KX, 1, m.status, s);
    else
      rc = tc_gemm_products(q.Rh != nullptr ? q.Rh + (size_t)t * l.BP * l.NP : m.X, m.W, m.partial, l.BP, (int)l.KX, l.NP, l.ns_z,
                           l.nt_z, m.status, s);
    if (rc != RINGRNN_OK) return rc;
    forward_row(p.activation, q, t, s);
    RINGRNN_CUDA_TRY(cudaGetLastError());
  }
  return RINGRNN_OK;
}

}  // namespace

int stepwise_forward(const RingRnnFwdArgs& a, const DevProblem& dp, cudaStream_t s) {
  const RingRnnProblem& p = a.p;
  const SwLayout l = sw_layout(p);
  if (a.workspace == nullptr || a.workspace_bytes < stepwise_fwd_workspace_bytes(p)) return RINGRNN_ERR_WORKSPACE;
  if ((reinterpret_cast<uintptr_t>(a.workspace) & 255) != 0) return RINGRNN_ERR_WORKSPACE;
  const bool train = a.saved != nullptr;
  if (train && (a.saved_bytes < stepwise_saved_bytes(p) || (reinterpret_cast<uintptr_t>(a.saved) & 255) != 0))
    return RINGRNN_ERR_WORKSPACE;
  char* w = static_cast<char*>(a.workspace);
  SwFwdBuffers m;
  m.status = a.status != nullptr ? a.status : reinterpret_cast<int*>(w);
  w += 1024;
  m.W = reinterpret_cast<__nv_bfloat16*>(w);
  w += align_up((size_t)l.NP * l.KX * 2, 1024);
  m.X = reinterpret_cast<__nv_bfloat16*>(w);
  w += x_bytes(l);
  m.state = reinterpret_cast<float*>(w);
  w += align_up((size_t)l.BP * l.NP * 4, 1024);
  m.rowsum = reinterpret_cast<float*>(w);
  w += align_up((size_t)l.BP * 4, 1024);
  m.partial = reinterpret_cast<float*>(w);
  if (a.status == nullptr) RINGRNN_CUDA_TRY(cudaMemsetAsync(m.status, 0, sizeof(int), s));
  const int K = train ? sw_ckpt_interval(p) : 0;
  if (K > 0)  // checkpoint 0 is the initial state
    RINGRNN_CUDA_TRY(cudaMemcpyAsync(a.saved, p.r_init, ckpt_slot(p), cudaMemcpyDeviceToDevice, s));
  const int rc = prepare_forward(p, dp, l, m, s);
  if (rc != RINGRNN_OK) return rc;
  SwFwd q;
  memset(&q, 0, sizeof(q));
  q.T = p.T;
  q.r_init = p.r_init;
  if (train && K == 0) {
    q.Rh = static_cast<__nv_bfloat16*>(a.saved);
    q.Dh = reinterpret_cast<__nv_bfloat16*>(static_cast<char*>(a.saved) + align_up((size_t)(p.T + 1) * l.BP * l.NP * 2, 1024));
  }
  q.ckpt = K > 0 ? static_cast<float*>(a.saved) : nullptr;
  q.ckpt_every = K;
  q.hist = a.bump_history; q.final_state = a.final_state;
  q.dec_x = a.dec_x; q.dec_y = a.dec_y; q.dec_ta = a.dec_ta; q.dec_u = a.dec_u; q.dec_v = a.dec_v;
  return run_forward(p, dp, l, m, q, s);
}

int stepwise_backward(const RingRnnBwdArgs& a, const DevProblem& dp, cudaStream_t s) {
  const RingRnnProblem& p = a.p;
  const SwLayout l = sw_layout(p);
  if (a.workspace == nullptr || a.workspace_bytes < stepwise_bwd_workspace_bytes(p)) return RINGRNN_ERR_WORKSPACE;
  if ((reinterpret_cast<uintptr_t>(a.workspace) & 255) != 0) return RINGRNN_ERR_WORKSPACE;
  if (a.saved == nullptr || a.saved_bytes < stepwise_saved_bytes(p) || (reinterpret_cast<uintptr_t>(a.saved) & 255) != 0)
    return RINGRNN_ERR_WORKSPACE;
  const int K = sw_ckpt_interval(p), Tk = K > 0 ? K : p.T;  // steps of one stretch
  const size_t w_bytes = align_up((size_t)l.KX * l.NP * 2, 1024), dw_bytes = align_up((size_t)l.NP * l.KX * 4, 1024);
  char* w = static_cast<char*>(a.workspace);
  auto take = [&w](size_t bytes) { char* at = w; w += bytes; return at; };
  int* scratch_status = reinterpret_cast<int*>(take(1024));
  int* status = a.status != nullptr ? a.status : scratch_status;
  __nv_bfloat16* WstT = reinterpret_cast<__nv_bfloat16*>(take(w_bytes));
  __nv_bfloat16* Delta = reinterpret_cast<__nv_bfloat16*>(take(align_up((size_t)Tk * l.BP * l.NP * 2, 1024)));
  float* g = reinterpret_cast<float*>(take(align_up((size_t)l.BP * l.NP * 4, 1024)));
  float* sum_delta = reinterpret_cast<float*>(take(align_up((size_t)l.BP * 4, 1024)));
  float* zpart = reinterpret_cast<float*>(take(z_bytes(l, false)));
  __nv_bfloat16* Xall = reinterpret_cast<__nv_bfloat16*>(take(align_up((size_t)Tk * l.BP * l.KX * 2, 1024)));
  float* dwpart = reinterpret_cast<float*>(take(align_up((size_t)dw_splits(l, Tk) * l.NP * l.KX * 4, 1024)));
  float* dWst = reinterpret_cast<float*>(take(dw_bytes));
  float* raw = reinterpret_cast<float*>(take(align_up((size_t)p.N * p.N * 4, 1024)));
  SwFwdBuffers m;
  memset(&m, 0, sizeof(m));
  char* stretch = nullptr;
  float* dWst_stretch = nullptr;
  if (K > 0) {
    m.W = reinterpret_cast<__nv_bfloat16*>(take(w_bytes));
    m.X = reinterpret_cast<__nv_bfloat16*>(take(x_bytes(l)));
    m.state = reinterpret_cast<float*>(take(align_up((size_t)l.BP * l.NP * 4, 1024)));
    m.rowsum = reinterpret_cast<float*>(take(align_up((size_t)l.BP * 4, 1024)));
    m.partial = zpart;
    m.status = status;
    stretch = take(every_step_bytes(l, K));
    dWst_stretch = reinterpret_cast<float*>(take(dw_bytes));
  }
  if (a.status == nullptr) RINGRNN_CUDA_TRY(cudaMemsetAsync(status, 0, sizeof(int), s));

  const SwCols cols = cols_of(dp);
  {
    LaunchScope ls(K_PREP, s);
    sw_prep_transposed_kernel<<<dim3(l.NP / 32, l.NP / 32, l.blocks), 256, 0, s>>>(p.Wo, dp.Wa, cols, p.J1, p.N, l.NP, WstT);
  }
  RINGRNN_CUDA_TRY(cudaGetLastError());
  if (K > 0) {
    const int rc = prepare_forward(p, dp, l, m, s);
    if (rc != RINGRNN_OK) return rc;
  }
  if (a.grad_A != nullptr)
    RINGRNN_CUDA_TRY(cudaMemsetAsync(a.grad_A, 0, sizeof(float) * (size_t)p.B * p.T * p.a_dim, s));

  // With checkpoints the stretches of K steps are taken last to first: each is recomputed from its fp32 state, then run in
  // reverse from the carry the later stretch left in g, and its weight gradients are added to the total.
  const int n_ck = (p.T + Tk - 1) / Tk;
  for (int c = n_ck - 1; c >= 0; --c) {
    const int t0 = c * Tk, Tc = p.T - t0 < Tk ? p.T - t0 : Tk;
    char* kept = K > 0 ? stretch : static_cast<char*>(const_cast<void*>(a.saved));
    __nv_bfloat16* Rh = reinterpret_cast<__nv_bfloat16*>(kept);
    __nv_bfloat16* Dh = reinterpret_cast<__nv_bfloat16*>(kept + align_up((size_t)(Tc + 1) * l.BP * l.NP * 2, 1024));
    if (K > 0) {
      SwFwd f;
      memset(&f, 0, sizeof(f));
      f.T = Tc; f.t0 = t0;
      f.r_init = static_cast<const float*>(a.saved) + (size_t)c * p.B * p.N;
      f.Rh = Rh; f.Dh = Dh;
      const int rc = run_forward(p, dp, l, m, f, s);
      if (rc != RINGRNN_OK) return rc;
    }
    SwBwd q;
    memset(&q, 0, sizeof(q));
    q.B = p.B; q.T = Tc; q.N = p.N; q.NP = l.NP; q.BP = l.BP; q.a_dim = p.a_dim; q.nsplit = l.ns_z;
    q.t0 = t0; q.T_total = p.T;
    q.resume = c != n_ck - 1;
    q.grad_r_init = c == 0 ? a.grad_r_init : nullptr;
    q.vec = p.N % 4 == 0 && aligned16(a.grad_output) && aligned16(q.grad_r_init);
    q.KX = l.KX; q.J0 = p.J0; q.alpha = p.alpha;
    q.A = p.A; q.grad_output = a.grad_output;
    q.coef_x = a.coef_x; q.coef_y = a.coef_y; q.coef_s = a.coef_s; q.dec_u = a.dec_u; q.dec_v = a.dec_v;
    q.Rh = Rh; q.Dh = Dh; q.partial = zpart; q.g = g; q.sum_delta = sum_delta; q.Delta = Delta;
    q.grad_A = a.grad_A; q.cols = cols;
    {
      LaunchScope ls(K_BWD, s);
      RINGRNN_CUDA_TRY(launch_row(sw_backward_row_kernel<false>, l.BP, l.NP, s, q, -1, Tc - 1));
    }
    for (int t = Tc - 1; t >= 0; --t) {
      // Z_t[BP, KX] = delta_t[BP, NP] x WstT[KX, NP]^T
      const int rc = tc_gemm_products(Delta + (size_t)t * l.BP * l.NP, WstT, zpart, l.BP, (int)l.KX, l.NP, l.ns_z, l.nt_z, status, s);
      if (rc != RINGRNN_OK) return rc;
      LaunchScope ls(K_BWD, s);
      RINGRNN_CUDA_TRY(q.grad_A != nullptr ? launch_row(sw_backward_row_kernel<true>, l.BP, l.NP, s, q, t, t - 1)
                                           : launch_row(sw_backward_row_kernel<false>, l.BP, l.NP, s, q, t, t - 1));
    }
    {
      LaunchScope ls(K_PREP, s);
      sw_build_xall_kernel<<<dim3(l.BP, Tc < MAX_GRID_Y ? Tc : MAX_GRID_Y), row_threads(l.NP), 0, s>>>(Rh, p.A, cols, p.B, Tc, t0, p.T, p.a_dim,
                                                                                                       l.NP, l.BP, l.KX, Xall);
    }
    RINGRNN_CUDA_TRY(cudaGetLastError());
    // dWst[NP, KX] = Delta^T [NP, Tc*BP] x Xall [Tc*BP, KX]
    const bool first = c == n_ck - 1;
    const int rc = tc_gemm(1, Delta, Xall, dwpart, first ? dWst : dWst_stretch, l.NP, (int)l.KX, (long long)Tc * l.BP,
                           dw_splits(l, Tc), status, s);
    if (rc != RINGRNN_OK) return rc;
    if (!first) {
      LaunchScope ls(K_REDUCE, s);
      sw_accumulate_kernel<<<592, 256, 0, s>>>(dWst, dWst_stretch, (size_t)l.NP * l.KX);
      RINGRNN_CUDA_TRY(cudaGetLastError());
    }
  }
  const size_t NN = (size_t)p.N * p.N;
  RINGRNN_CUDA_TRY(cudaMemsetAsync(a.grad_Wa, 0, sizeof(float) * (size_t)p.a_dim * NN, s));
  {
    LaunchScope ls(K_REDUCE, s);
    sw_unpack_dw_kernel<<<296, 256, 0, s>>>(dWst, p.N, l.NP, l.KX, p.J1, cols, a.grad_Wo, a.grad_Wa, raw);
  }
  RINGRNN_CUDA_TRY(cudaGetLastError());
  if (a.grad_J != nullptr) {
    // the dW split-K partials are dead after the reduction inside tc_gemm: their storage serves as scratch
    const int rc = launch_grad_j(raw, p.Wo, NN, a.grad_J, reinterpret_cast<double*>(dwpart), s);
    if (rc != RINGRNN_OK) return rc;
  }
  return RINGRNN_OK;
}

}  // namespace ringrnn
