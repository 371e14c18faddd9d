// fp32 mode, recurrent kernels for weights that fit the shared memory of a thread-block cluster.
//
// A cluster of C CTAs owns a tile of 8*NO samples for the whole sequence.  CTA q keeps rows [q*NC, q*NC + NC) of all
// matrices in shared memory, fp32, for all T steps, and holds the full state of the tile; per step it forms its NC neurons
// of  re = sum_m c_m (W_m r)  on the CUDA cores and stores its part of the new state into every CTA's next state buffer
// (distributed shared memory), one cluster barrier per step.  J0 and J1 are folded into the first matrix (J1*Wo + J0).
// What bounds it (N = 250, B = 200, cycles of a forward step of 11.5 K): the products 5.5 K (3.1 K of it FMA issue, the rest
// 16-byte shared-memory loads of four wavefronts each), summing and activation with the stores into eight CTAs 1.4 K,
// global memory behind the arrival 1.8 K, the barrier 0.9 K, decode sums 1.8 K.  One CTA per 16 samples with the weights read
// through L2 took 75 us per forward and 190 us per reverse step there; now 5.8 and 6.1.
//
// Phase 1 (products): the K range is dealt to 8 warps x 4 lane groups; a thread holds 4 neurons x 8*OP samples, so one
// 16-byte weight load and 2*OP 16-byte state loads feed 32*OP FMAs (packed pairs).  The matrices are mixed in registers,
// which leaves one value per neuron and sample to be summed over the 32 K slices: over the lane groups with shuffles, over
// the warps through shared memory, in a fixed order.
// Phase 2: a thread per (neuron, 2 samples) sums the eight partials, applies the step's arithmetic, writes global memory
// (consecutive lanes = consecutive neurons) and the state buffers.
//
//   MODE 0  forward.  Also writes F'(re) when asked to (dact), which is what the reverse kernel needs.
//   MODE 1  F'(re) of every step from a given history: the same products without the recurrence, the time range split over
//           blockIdx.y.
//   MODE 2  reverse time: state = delta_t, matrices transposed.
#pragma once

#include "ringrnn_common.cuh"
#include "tc_ptx.cuh"

namespace ringrnn {
namespace fc {

constexpr int THREADS = 256;

struct Shape {
  int C, NC, NO, NP;  // CTAs per cluster, neurons per CTA (multiple of 32), sample octets, N padded to 32
  int tiles;          // ceil(B / (8*NO))
};

struct Args {
  DevProblem p;
  Shape sh;
  float* hist;           // MODE 0: out or nullptr; 1, 2: in  [T,B,N]
  float* dact;           // [T,B,N] F'(re): MODE 0 out or nullptr, 1 out, 2 in (may be delta: the same thread reads, then writes)
  // forward
  float* dec_x;          // [B,T] or nullptr
  float* dec_y;
  float* dec_ta;
  float* final_state;    // [B,N] or nullptr
  // reverse
  const float* grad_output;
  const float* coef_x;
  const float* coef_y;
  const float* coef_s;
  const float* dec_u;
  const float* dec_v;
  float* delta;          // [T,B,N]
  float* grad_r_init;
  float* dA_part;        // [C][n_mat-1][B][T] or nullptr
};

// shared memory, in floats
struct Off {
  int w, s, part, sc, uv, cf, g, rb, dp, total;
};
__host__ __device__ inline Off offsets(const Shape& h, int n_mat, int mode) {
  Off o;
  int at = 0;
  o.w = at; at += n_mat * h.NP * h.NC;          // [m][k][perm(neuron)]
  o.s = at; at += 2 * h.NO * 8 * h.NP;          // [2][quad][k][4]
  o.part = at; at += 8 * h.NO * 8 * h.NC;       // [warp][quad][neuron][4]
  o.sc = at; at += 2 * n_mat * h.NO * 8;        // [2][m][sample]
  o.uv = at; at += mode != 1 ? 2 * h.NP : 0;    // decode vectors
  o.cf = at; at += mode == 2 ? 3 * h.NO * 8 : 0;
  o.g = at; at += mode == 2 ? h.NO * 8 * h.NC : 0;   // carry / g of this CTA's neurons  [quad][neuron][4]
  o.rb = at; at += mode == 2 ? h.NO * 8 * h.NC : 0;  // r_{t-1} likewise (dL/dA)
  o.dp = at; at += mode == 2 ? 8 * n_mat * h.NO * 8 : 0;  // dL/dA sums per warp
  o.total = at;
  return o;
}

__device__ __forceinline__ unsigned long long pk(float a, float b) {
  unsigned long long r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
  return r;
}
__device__ __forceinline__ void upk(unsigned long long v, float& a, float& b) {
  asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v));
}
__device__ __forceinline__ unsigned long long fma2(unsigned long long a, unsigned long long b, unsigned long long c) {
  unsigned long long d;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
  return d;
}
__device__ __forceinline__ float4 ld4(const float* p) { return *reinterpret_cast<const float4*>(p); }

// Phase 1 for one neuron group of 32 and OP octets starting at octet o0: partial sums of the mixed product into part[].
template <int OP, bool WANT_DA>
__device__ __forceinline__ void products(const Args& a, const Off& of, float* sm, int cur, int grp, int o0, int warp, int lane) {
  const Shape& h = a.sh;
  const int slice = lane >> 3, nl = lane & 7;
  const float* s = sm + of.s + cur * (h.NO * 8 * h.NP);
  const float* sc = sm + of.sc + cur * (a.p.n_mat * h.NO * 8);
  unsigned long long re[4][4 * OP];
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int b = 0; b < 4 * OP; ++b) re[i][b] = 0ull;
  for (int m = 0; m < a.p.n_mat; ++m) {
    unsigned long long acc[4][4 * OP];
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int b = 0; b < 4 * OP; ++b) acc[i][b] = 0ull;
    const float* w = sm + of.w + (size_t)m * h.NP * h.NC + grp * 32 + nl * 4;
#pragma unroll 2
    for (int k = warp * 4 + slice; k < h.NP; k += 32) {
      const float4 wv = ld4(w + k * h.NC);
      const unsigned long long w2[4] = {pk(wv.x, wv.x), pk(wv.y, wv.y), pk(wv.z, wv.z), pk(wv.w, wv.w)};
#pragma unroll
      for (int q = 0; q < 2 * OP; ++q) {
        const float4 sv = ld4(s + ((o0 * 2 + q) * h.NP + k) * 4);
        const unsigned long long s0 = pk(sv.x, sv.y), s1 = pk(sv.z, sv.w);
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          acc[i][2 * q] = fma2(w2[i], s0, acc[i][2 * q]);
          acc[i][2 * q + 1] = fma2(w2[i], s1, acc[i][2 * q + 1]);
        }
      }
    }
    if (WANT_DA && m > 0) {
      // dL/dA: sum over this thread's neurons of r_{t-1} * (its share of Z_m), then over the warp, fixed order
      float v[8 * OP];
#pragma unroll
      for (int b = 0; b < 8 * OP; ++b) v[b] = 0.f;
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int q = 0; q < 2 * OP; ++q) {
          const float4 r = ld4(sm + of.rb + ((o0 * 2 + q) * h.NC + grp * 32 + i * 8 + nl) * 4);
          float x0, x1, x2, x3;
          upk(acc[i][2 * q], x0, x1);
          upk(acc[i][2 * q + 1], x2, x3);
          v[4 * q] = fmaf(r.x, x0, v[4 * q]);
          v[4 * q + 1] = fmaf(r.y, x1, v[4 * q + 1]);
          v[4 * q + 2] = fmaf(r.z, x2, v[4 * q + 2]);
          v[4 * q + 3] = fmaf(r.w, x3, v[4 * q + 3]);
        }
#pragma unroll
      for (int b = 0; b < 8 * OP; ++b) {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) v[b] += __shfl_xor_sync(0xffffffffu, v[b], o);
        if (lane == 0) {
          float* d = sm + of.dp + (warp * a.p.n_mat + m) * (h.NO * 8) + o0 * 8 + b;
          *d = grp == 0 ? v[b] : *d + v[b];
        }
      }
    }
#pragma unroll
    for (int q = 0; q < 2 * OP; ++q) {
      const float4 cv = m == 0 ? make_float4(1.f, 1.f, 1.f, 1.f) : ld4(sc + m * (h.NO * 8) + (o0 * 2 + q) * 4);
      const unsigned long long c0 = pk(cv.x, cv.y), c1 = pk(cv.z, cv.w);
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        re[i][2 * q] = fma2(c0, acc[i][2 * q], re[i][2 * q]);
        re[i][2 * q + 1] = fma2(c1, acc[i][2 * q + 1], re[i][2 * q + 1]);
      }
    }
  }
  // over the four K slices of the warp: afterwards the lane holds neuron 8*slice + nl of the group
  float* part = sm + of.part + warp * (h.NO * 8 * h.NC);
#pragma unroll
  for (int q = 0; q < 2 * OP; ++q) {
    float v[4][4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      upk(re[i][2 * q], v[i][0], v[i][1]);
      upk(re[i][2 * q + 1], v[i][2], v[i][3]);
    }
    float k2[2][4], out[4];
    const bool up = lane & 16;
#pragma unroll
    for (int i = 0; i < 2; ++i)
#pragma unroll
      for (int b = 0; b < 4; ++b) {
        const float send = up ? v[i][b] : v[i + 2][b], keep = up ? v[i + 2][b] : v[i][b];
        k2[i][b] = keep + __shfl_xor_sync(0xffffffffu, send, 16);
      }
    const bool up2 = lane & 8;
#pragma unroll
    for (int b = 0; b < 4; ++b) {
      const float send = up2 ? k2[0][b] : k2[1][b], keep = up2 ? k2[1][b] : k2[0][b];
      out[b] = keep + __shfl_xor_sync(0xffffffffu, send, 8);
    }
    // i = 2*bit4 + bit3 = slice, the neuron's index within the permuted group of four
    *reinterpret_cast<float4*>(part + ((o0 * 2 + q) * h.NC + grp * 32 + slice * 8 + nl) * 4) =
        make_float4(out[0], out[1], out[2], out[3]);
  }
}

template <int MODE, int ACT>
__global__ void __launch_bounds__(THREADS, 1) cluster_kernel(const __grid_constant__ Args a) {
  extern __shared__ __align__(16) float sm[];
  const Shape& h = a.sh;
  const DevProblem& p = a.p;
  const Off of = offsets(h, p.n_mat, MODE);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int rank = h.C > 1 ? (int)tc::cluster_ctarank() : 0;
  const int cluster = blockIdx.x / h.C, n_clusters = gridDim.x / h.C;
  const int N = p.N, NP = h.NP, NC = h.NC, BT = 8 * h.NO, quads = 2 * h.NO;
  const int i0 = rank * NC;
  const bool want_dA = MODE == 2 && a.dA_part != nullptr;
  const bool want_dec = MODE == 0 && (a.dec_x != nullptr || a.dec_y != nullptr || a.dec_ta != nullptr);
  const uint32_t s_addr = tc::smem_u32(sm + of.s);

  // weights: position p of a group of 32 holds neuron (p % 4) * 8 + p / 4, so that a thread's four neurons are one 16-byte
  // load and its results land in different banks
  for (int m = 0; m < p.n_mat; ++m) {
    const float* W = m == 0 ? p.Wo : p.Wa + (size_t)active_col(p, m - 1) * N * N;
    float* dst = sm + of.w + (size_t)m * NP * NC;
    for (int idx = threadIdx.x; idx < NP * NC; idx += THREADS) {
      int k, n;  // consecutive threads read consecutive addresses
      if (MODE == 2) { k = idx / NC; n = idx % NC; }
      else { n = idx / NP; k = idx % NP; }
      const int i = i0 + n;
      float v = 0.f;
      if (i < N && k < N) {
        v = MODE == 2 ? W[(size_t)k * N + i] : W[(size_t)i * N + k];
        if (m == 0) v = fmaf(p.J1, v, p.J0);
      }
      const int nn = n & 31;
      dst[k * NC + (n & ~31) + (nn & 7) * 4 + (nn >> 3)] = v;
    }
  }
  if (MODE != 1)
    for (int idx = threadIdx.x; idx < 2 * NP; idx += THREADS) {
      const int k = idx % NP;
      sm[of.uv + idx] = a.dec_u != nullptr && k < N ? (idx < NP ? a.dec_u : a.dec_v)[k] : 0.f;
    }
  // the state rows beyond N are never written again: zero in both buffers
  for (int idx = threadIdx.x; idx < 2 * quads * NP * 4; idx += THREADS) sm[of.s + idx] = 0.f;
  __syncthreads();
  if (h.C > 1) {
    tc::cluster_arrive();
    tc::cluster_wait();
  }

  // MODE 1: this block row's share of the time range
  const int t_lo = MODE == 1 ? (int)((long long)p.T * blockIdx.y / gridDim.y) : 0;
  const int t_hi = MODE == 1 ? (int)((long long)p.T * (blockIdx.y + 1) / gridDim.y) : p.T;

  // action signal of step t: one value per thread fetched ahead (the whole of it with up to 256 / BT columns)
  auto fetch_scalar = [&](int b0, int t, int idx) {
    const int m = 1 + idx / BT, b = idx % BT;
    return b0 + b < p.B ? __ldg(p.A + ((size_t)(b0 + b) * p.T + t) * p.a_dim + active_col(p, m - 1)) : 0.f;
  };
  const int n_sc = (p.n_mat - 1) * BT;
  auto put_scalars = [&](int b0, int t, int buf, float ahead) {
    float* dst = sm + of.sc + (buf * p.n_mat + 1) * BT;
    if ((int)threadIdx.x < n_sc) dst[threadIdx.x] = ahead;
    for (int idx = threadIdx.x + THREADS; idx < n_sc; idx += THREADS) dst[idx] = fetch_scalar(b0, t, idx);
  };
  // Two samples of neuron row k into buffer `buf` of every CTA of the cluster.  Neighbouring lanes hold the two halves of a
  // quad: they put them together, so that a store carries 16 bytes, and take half of the destinations each.
  uint32_t peer[4];
#pragma unroll
  for (int c = 0; c < 4; ++c) {
    const int dst = c + (lane & 1) * (h.C / 2);
    peer[c] = h.C > 1 && c < h.C / 2 ? tc::mapa(s_addr, (uint32_t)dst) : 0u;
  }
  auto store_state = [&](int buf, int pair, int k, float2 v) {  // whole warps call it
    const uint32_t off = (uint32_t)(((buf * quads + pair / 2) * NP + k) * 16);
    if (h.C == 1) {
      *reinterpret_cast<float2*>(reinterpret_cast<uint8_t*>(sm + of.s) + off + (pair & 1) * 8) = v;
    } else {
      const float2 w = make_float2(__shfl_xor_sync(0xffffffffu, v.x, 1), __shfl_xor_sync(0xffffffffu, v.y, 1));
      const float2 lo = (lane & 1) ? w : v, hi = (lane & 1) ? v : w;
#pragma unroll
      for (int c = 0; c < 4; ++c)
        if (c < h.C / 2)
          tc::st_cluster_v4(peer[c] + off, __float_as_uint(lo.x), __float_as_uint(lo.y), __float_as_uint(hi.x),
                            __float_as_uint(hi.y));
    }
  };
  auto cluster_sync = [&]() {
    if (h.C > 1) {
      tc::cluster_arrive();
      tc::cluster_wait();
    } else {
      __syncthreads();
    }
  };

  for (int tile = cluster; tile < h.tiles; tile += n_clusters) {
    const int b0 = tile * BT;
    int cur = 0;
    // item = (4 samples, 16 neurons), two samples per lane; a warp's first two are handled from registers fetched ahead
    const int n_items = quads * (NC / 16);
    auto pair_of = [&](int it) { return 2 * (it % quads) + (lane & 1); };
    auto n_of = [&](int it) { return (it / quads) * 16 + (lane >> 1); };
    auto items = [&](auto&& f) {
      for (int it = warp; it < n_items; it += 8) f(pair_of(it), n_of(it));
    };
    auto load2 = [&](const float* base, size_t row_stride, int pair, int i) {  // samples 2*pair, 2*pair + 1 of neuron i
      float2 v = make_float2(0.f, 0.f);
      const int b = b0 + 2 * pair;
      if (i < N) {
        const float* src = base + (size_t)b * row_stride + i;
        if (b < p.B) v.x = __ldg(src);
        if (b + 1 < p.B) v.y = __ldg(src + row_stride);
      }
      return v;
    };
    auto load2_own = [&](const float* base, int pair, int i) {  // of a tensor this thread may overwrite there: not a read-only load
      float2 v = make_float2(0.f, 0.f);
      const int b = b0 + 2 * pair;
      if (i < N) {
        const float* src = base + (size_t)b * N + i;
        if (b < p.B) v.x = src[0];
        if (b + 1 < p.B) v.y = src[N];
      }
      return v;
    };
    auto save2 = [&](float* base, size_t row_stride, int pair, int i, float2 v) {
      const int b = b0 + 2 * pair;
      if (i < N) {
        float* dst = base + (size_t)b * row_stride + i;
        if (b < p.B) dst[0] = v.x;
        if (b + 1 < p.B) dst[row_stride] = v.y;
      }
    };
    // this thread's two values of a [quad][neuron][4] buffer of this CTA's neurons
    auto own = [&](int off, int pair, int n) { return reinterpret_cast<float2*>(sm + off + ((pair / 2) * NC + n) * 4 + (pair & 1) * 2); };
    const size_t slab = (size_t)p.B * N;
    const bool has_coef = MODE == 2 && a.coef_x != nullptr;
    auto fetch_coef = [&](int t) {  // 3*BT <= 96 values, one per thread
      if (!has_coef || (int)threadIdx.x >= 3 * BT) return 0.f;
      const int c = threadIdx.x / BT, b = threadIdx.x % BT;
      const float* src = c == 0 ? a.coef_x : c == 1 ? a.coef_y : a.coef_s;
      return b0 + b < p.B ? __ldg(src + (size_t)(b0 + b) * p.T + t) : 0.f;
    };
    // reverse: what g_t and delta_t need from global memory: F'(re_t), the caller's gradient, r_t (for its sign)
    struct Ahead { float2 d, go, r; };
    auto fetch = [&](int t, int pair, int n) {
      Ahead x;
      x.d = load2_own(a.dact + t * slab, pair, i0 + n);
      x.go = a.grad_output != nullptr ? load2(a.grad_output + t * slab, N, pair, i0 + n) : make_float2(0.f, 0.f);
      x.r = has_coef ? load2(a.hist + t * slab, N, pair, i0 + n) : make_float2(0.f, 0.f);
      return x;
    };
    Ahead ahead[2];
    auto fetch_ahead = [&](int t) {
#pragma unroll
      for (int j = 0; j < 2; ++j) {
        const int it = warp + 8 * j;
        if (it < n_items) ahead[j] = fetch(t, pair_of(it), n_of(it));
      }
    };
    // reverse: g_t from the carry, delta_t into buffer `buf`; returned so that it can be stored behind the exchange
    auto produce = [&](int buf, int pair, int n, const Ahead& x) {
      const int i = i0 + n;
      float2* gp = own(of.g, pair, n);
      float2 g = *gp;
      g.x += x.go.x; g.y += x.go.y;
      if (has_coef && i < N) {
        const float u = sm[of.uv + i], v = sm[of.uv + NP + i];
        const float* cf = sm + of.cf + 2 * pair;
        auto sg = [](float r) { return r > 0.f ? 1.f : r < 0.f ? -1.f : 0.f; };
        g.x += cf[0] * u + cf[BT] * v + cf[2 * BT] * sg(x.r.x);
        g.y += cf[1] * u + cf[BT + 1] * v + cf[2 * BT + 1] * sg(x.r.y);
      }
      *gp = g;
      const float2 d = make_float2(x.d.x * p.alpha * g.x, x.d.y * p.alpha * g.y);
      if (i < NP) store_state(buf, pair, i, d);
      return d;
    };
    auto produce_all = [&](int t, int buf) {
      float2 d[2];
#pragma unroll
      for (int j = 0; j < 2; ++j) {
        const int it = warp + 8 * j;
        if (it < n_items) d[j] = produce(buf, pair_of(it), n_of(it), ahead[j]);
      }
      for (int it = warp + 16; it < n_items; it += 8) {
        const int pair = pair_of(it), n = n_of(it);
        save2(a.delta + t * slab, N, pair, i0 + n, produce(buf, pair, n, fetch(t, pair, n)));
      }
      if (h.C > 1) tc::cluster_arrive();  // what follows need not be waited for by the peers
#pragma unroll
      for (int j = 0; j < 2; ++j) {
        const int it = warp + 8 * j;
        if (it < n_items) save2(a.delta + t * slab, N, pair_of(it), i0 + n_of(it), d[j]);
      }
      if (h.C > 1) tc::cluster_wait();
      else __syncthreads();
    };

    if (MODE == 0) {
      items([&](int pair, int n) {
        if (i0 + n < NP) store_state(0, pair, i0 + n, load2(p.r_init, N, pair, i0 + n));
      });
      put_scalars(b0, 0, 0, (int)threadIdx.x < n_sc ? fetch_scalar(b0, 0, threadIdx.x) : 0.f);
      cluster_sync();
    } else if (MODE == 2) {
      items([&](int pair, int n) { *own(of.g, pair, n) = make_float2(0.f, 0.f); });
      const float cf = fetch_coef(p.T - 1);
      if (has_coef && (int)threadIdx.x < 3 * BT) sm[of.cf + threadIdx.x] = cf;
      put_scalars(b0, p.T - 1, 0, (int)threadIdx.x < n_sc ? fetch_scalar(b0, p.T - 1, threadIdx.x) : 0.f);
      fetch_ahead(p.T - 1);
      __syncthreads();
      produce_all(p.T - 1, 0);
    }

    for (int step = t_lo; step < t_hi; ++step) {
      const int t = MODE == 2 ? p.T - 1 - step : step;
      if (MODE == 1) {  // the state before step t, straight from the history
        const float* prev = t == 0 ? p.r_init : a.hist + (size_t)(t - 1) * slab;
        __syncthreads();
        for (int it = warp; it < 2 * quads * (NP / 32); it += 8) {
          const int pair = it % (2 * quads), k = (it / (2 * quads)) * 32 + lane;
          *reinterpret_cast<float2*>(sm + of.s + ((pair / 2) * NP + k) * 4 + (pair & 1) * 2) = load2(prev, N, pair, k);
        }
        put_scalars(b0, t, 0, (int)threadIdx.x < n_sc ? fetch_scalar(b0, t, threadIdx.x) : 0.f);
        __syncthreads();
      }
      // the next step's inputs, in flight under the products
      const int tn = MODE == 2 ? t - 1 : t + 1;
      const bool more = MODE != 1 && tn >= 0 && tn < p.T;
      const float sc_ahead = more && (int)threadIdx.x < n_sc ? fetch_scalar(b0, tn, threadIdx.x) : 0.f;
      const float cf_ahead = more ? fetch_coef(tn) : 0.f;
      if (MODE == 2 && more) fetch_ahead(tn);
      if (want_dA) {
        const float* prev = t == 0 ? p.r_init : a.hist + (size_t)(t - 1) * slab;
        items([&](int pair, int n) { *own(of.rb, pair, n) = load2(prev, N, pair, i0 + n); });
        __syncthreads();
      }
      for (int grp = 0; grp < NC / 32; ++grp) {
        int o = 0;
        if (MODE == 2 && want_dA) {
          for (; o < h.NO; ++o) products<1, true>(a, of, sm, cur, grp, o, warp, lane);
        } else {
          for (; o + 2 <= h.NO; o += 2) products<2, false>(a, of, sm, cur, grp, o, warp, lane);
          if (o < h.NO) products<1, false>(a, of, sm, cur, grp, o, warp, lane);
        }
      }
      if (more) {
        put_scalars(b0, tn, cur ^ 1, sc_ahead);
        if (has_coef && (int)threadIdx.x < 3 * BT) sm[of.cf + threadIdx.x] = cf_ahead;
      }
      __syncthreads();
      auto total = [&](int pair, int n) {
        float2 z = make_float2(0.f, 0.f);
#pragma unroll
        for (int w = 0; w < 8; ++w) {
          const float2 x = *own(of.part + w * (h.NO * 8 * NC), pair, n);
          z.x += x.x; z.y += x.y;
        }
        return z;
      };
      const float beta = 1.f - p.alpha;
      if (MODE == 2) {
        items([&](int pair, int n) {  // the carry, in place of g
          const float2 z = total(pair, n);
          float2* gp = own(of.g, pair, n);
          const float2 cv = make_float2(fmaf(beta, gp->x, z.x), fmaf(beta, gp->y, z.y));
          *gp = cv;
          if (t == 0 && a.grad_r_init != nullptr) save2(a.grad_r_init, N, pair, i0 + n, cv);
        });
        if (want_dA) {
          // sums over the warps of this CTA's neurons; the CTAs' parts are added up afterwards
          for (int idx = threadIdx.x; idx < n_sc; idx += THREADS) {
            const int m = 1 + idx / BT, b = idx % BT;
            float v = 0.f;
            for (int w = 0; w < 8; ++w) v += sm[of.dp + (w * p.n_mat + m) * BT + b];
            if (b0 + b < p.B) a.dA_part[(((size_t)rank * (p.n_mat - 1) + m - 1) * p.B + b0 + b) * p.T + t] = v;
          }
        }
        if (more) produce_all(tn, cur ^ 1);
        else cluster_sync();
        cur ^= 1;
      } else {
        auto advance = [&](int pair, int n, float2 z) {
          const int i = i0 + n;
          float2 r = make_float2(0.f, 0.f);
          if (i < N) {
            const float2 o = *reinterpret_cast<const float2*>(sm + of.s + ((cur * quads + pair / 2) * NP + i) * 4 + (pair & 1) * 2);
            r = make_float2(fmaf(p.alpha, act_fn<ACT>(z.x), beta * o.x), fmaf(p.alpha, act_fn<ACT>(z.y), beta * o.y));
          }
          if (i < NP) store_state(cur ^ 1, pair, i, r);
          return r;
        };
        auto record = [&](int pair, int n, float2 z, float2 r) {
          if (a.dact != nullptr)
            save2(a.dact + t * slab, N, pair, i0 + n, make_float2(act_grad<ACT>(z.x), act_grad<ACT>(z.y)));
          if (MODE == 0) {
            if (a.hist != nullptr) save2(a.hist + t * slab, N, pair, i0 + n, r);
            if (a.final_state != nullptr && t + 1 == p.T) save2(a.final_state, N, pair, i0 + n, r);
          }
        };
        float2 z[2], r[2];
#pragma unroll
        for (int j = 0; j < 2; ++j) {
          const int it = warp + 8 * j, pair = pair_of(it), n = n_of(it);
          if (it < n_items) {
            z[j] = total(pair, n);
            r[j] = MODE == 0 ? advance(pair, n, z[j]) : z[j];
          }
        }
        for (int it = warp + 16; it < n_items; it += 8) {
          const int pair = pair_of(it), n = n_of(it);
          const float2 zz = total(pair, n);
          record(pair, n, zz, MODE == 0 ? advance(pair, n, zz) : zz);
        }
        // global memory behind the arrival: the peers need not wait for these stores
        if (MODE == 0 && h.C > 1) tc::cluster_arrive();
#pragma unroll
        for (int j = 0; j < 2; ++j) {
          const int it = warp + 8 * j;
          if (it < n_items) record(pair_of(it), n_of(it), z[j], r[j]);
        }
        if (MODE == 0) {
          if (h.C > 1) tc::cluster_wait();
          else __syncthreads();
          cur ^= 1;
        }
      }
      if (want_dec) {
        // r_t is complete in this CTA's buffer: decode sums, four samples per warp, dealt over the cluster's warps
        for (int quad = rank + h.C * warp; quad < quads; quad += h.C * 8) {
          float v[12];
#pragma unroll
          for (int j = 0; j < 12; ++j) v[j] = 0.f;
#pragma unroll 4
          for (int k = lane; k < NP; k += 32) {
            const float4 r = ld4(sm + of.s + ((cur * quads + quad) * NP + k) * 4);
            const float u = sm[of.uv + k], w = sm[of.uv + NP + k];
            v[0] = fmaf(r.x, u, v[0]); v[1] = fmaf(r.y, u, v[1]); v[2] = fmaf(r.z, u, v[2]); v[3] = fmaf(r.w, u, v[3]);
            v[4] = fmaf(r.x, w, v[4]); v[5] = fmaf(r.y, w, v[5]); v[6] = fmaf(r.z, w, v[6]); v[7] = fmaf(r.w, w, v[7]);
            v[8] += fabsf(r.x); v[9] += fabsf(r.y); v[10] += fabsf(r.z); v[11] += fabsf(r.w);
          }
#pragma unroll
          for (int j = 0; j < 12; ++j)
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) v[j] += __shfl_xor_sync(0xffffffffu, v[j], o);
          float mine = v[0];  // lane j writes value j
#pragma unroll
          for (int j = 1; j < 12; ++j) mine = lane == j ? v[j] : mine;
          const int b = b0 + 4 * quad + (lane & 3);
          float* dst = lane < 4 ? a.dec_x : lane < 8 ? a.dec_y : a.dec_ta;
          if (lane < 12 && b < p.B && dst != nullptr) dst[(size_t)b * p.T + t] = mine;
        }
      }
    }
    if (MODE != 1) cluster_sync();  // nobody rewrites a state buffer that a peer still reads
    else __syncthreads();
  }
}

}  // namespace fc
}  // namespace ringrnn
