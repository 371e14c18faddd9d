// Recurrent kernels with neurons on the tensor-memory lanes (bf16 mode, N <= 512, up to two active action columns).
//
// The products of a step are taken as  D_m[neuron, sample] = W_m[128 neurons, NP] x r^T[NP, S samples]: the weights are the
// A operand and stay on the chip for the whole sequence, the state of S samples is the B operand.  Compared with samples on
// the lanes (tc_recurrent.cuh) a CTA may own as few as 16 samples, so a batch of 128 spreads over 8 SMs and one of 1024 over
// 64 clusters instead of 8, no weight byte moves inside the loop, and what a step costs is its latency chain alone:
// 32 or 64 small MMAs, one accumulator read of S/2 columns per thread, the activation, a store of the new state.
//
//   NP = 128: one CTA.  NP = 256: a cluster of two CTAs, CTA q owns neurons [128q, 128q+128) and stores its half of the new
//   state into both CTAs' operand buffers (16-byte asynchronous stores through distributed shared memory; the buffers alternate, so nobody waits
//   for a peer's MMAs: a peer that has sent r_t has finished the MMAs that read r_{t-2}).
//
//   NP = 512: a cluster of four, likewise, 16 samples per cluster.
//
// A operand.  Matrices that fit are kept in TENSOR MEMORY (128 lanes x NP/2 columns each): an MMA with a 16-column B operand
// is bound by fetching its A tile, 4 KB at 128 B/clk from shared memory against 8-16 cycles from tensor memory.  The rest
// of the three (where 64 samples per unit leave no columns; at NP = 512, 44 of the 96 K steps) are in shared memory,
// K-major, 128-byte swizzle.
// Global inhibition.  J0 * sum_j r_j joins the Wo product: J1 * (Yo + (J0/J1) * S) with S from an MMA whose A tile is
// constant along both dimensions, the same 16-column tile for every K step.  J0/J1 enters as up to three bf16 terms (24
// bits); one is enough for the usual J0 = -J1.
// B operand.  [NP rows = neurons] x [64 samples] bf16, 128 bytes per row, 128-byte swizzle ("MN-major"); an MMA reads the
// first S samples.  NP = 512, where shared memory is short: 16 samples, 32 bytes per row, 32-byte swizzle.  A thread owns a neuron, so it writes its new values as 16-byte pieces of a row.
//
// What it gives over tiles of 128 samples, training steps: N = 120 B = 128 T = 120 1274 -> 315 us (428 with the old host path),
// N = 256 B = 1024 T = 256 3390 -> 1200, N = 512 B = 64 T = 64 1464 -> 772; roll-out N = 120 B = 65536 T = 4000 65.0 -> 46.1 ms.
//
// Roles (128 + 256 U threads): warp 0 issues the MMAs, warp 1 allocates tensor memory, warp 2 stages the per-sample
// scalars (action signal, loss coefficients) eight steps at a time, the last 8 U warps are the epilogue: unit u has eight,
// warp w of them owns lanes 32 (w & 3).. and the half h = w >> 2 of the unit's samples (E = S/2 per thread).
// U = 2 units of S samples run side by side in a CTA, one unit's MMAs under the other's epilogue.  Unit u of the c-th of G
// clusters takes tiles c + G (u + U round), so that a last round of up to G tiles has one, and is faster, in every CTA.
#pragma once

#include "tc_recurrent.cuh"

namespace ringrnn {

struct LaneFwdParams {
  int B, T, N, BPs, n_ut, a_dim, colL, colR;  // n_ut = unit tiles of S samples; BPs = n_ut * S
  float J1, alpha;       // J1 = 1 and use_wo = 0 when J0/J1 cannot be formed
  int use_wo, n_const;   // n_const: bf16 terms of J0/J1
  float cterm[3];
  const float* Wo;       // [N,N]
  const float* WL;       // [N,N] or nullptr
  const float* WR;
  int w_vec;             // 16-byte loads of matrix rows are aligned (N a multiple of four and every matrix so aligned)
  int dec_vec;           // likewise 16-byte stores of four steps' decode sums
  const float* A;        // [B,T_total,a_dim]
  const float* r_init;   // [B,N]
  __nv_bfloat16* Rh;     // [T+1][NP][BPs] (slot 0 = r_init) or nullptr
  __nv_bfloat16* Dh;     // F'(re), private layout, T*NP*BPs elements
  uint32_t* Sg;          // sign / zero bits of r_t, private layout, T*NP*BPs/4 bytes
  float* hist;           // [T,B,N] or nullptr
  float* dec[4][3];      // [B][T] decode sums r.u, r.v, sum|r| over the neurons of each CTA; nullptr = not wanted
  const float* dec_u;    // [N]
  const float* dec_v;
  float* final_state;    // [B,N] or nullptr
  float* ckpt;           // as in TcFwdParams
  int ckpt_every;
  int t0, T_total;
  int* status;            // receives the code of an abandoned wait; polled by slow waits
  volatile int* host;     // pinned host word that receives it too, or nullptr
};

struct LaneBwdParams {
  int B, T, N, BPs, n_ut, a_dim, colL, colR;
  float J1, alpha;
  int use_wo, n_const;
  float cterm[3];
  const float* Wo;
  const float* WL;
  const float* WR;
  const float* A;
  const __nv_bfloat16* Rh;    // [T+1][NP][BPs] (read only for dA)
  const __nv_bfloat16* Dh;
  const uint32_t* Sg;
  const float* grad_output;   // [T_total,B,N] or nullptr
  const float* coef_x;        // [B,T_total] or nullptr
  const float* coef_y;
  const float* coef_s;
  const float* dec_u;
  const float* dec_v;
  __nv_bfloat16* DL;          // [T][3][NP][BPs]: delta, L*delta, R*delta
  float* grad_r_init;         // [B,N] or nullptr
  float* dA_part;             // [CL][2][T][BPs] or nullptr
  const float* carry_in;      // [B,N] or nullptr
  int t0, T_total;
  int* status;            // receives the code of an abandoned wait; polled by slow waits
  volatile int* host;     // pinned host word that receives it too, or nullptr
};

// samples per unit: 16, 32 or 64 (see lane_unit_samples); units: 1 or 2 per CTA
int lane_forward_launch(int act, int NP, int S, int units, const LaneFwdParams& p, cudaStream_t s);
int lane_backward_launch(int NP, int S, const LaneBwdParams& p, cudaStream_t s);

namespace lane {

using namespace tc;
using tcr::f32x2;
using tcr::fma2;
using tcr::mul2;
using tcr::pack_bf16x2;
using tcr::pk2;
using tcr::pk2u;
using tcr::upk2;

constexpr int CH = 8;  // steps whose scalars are staged at a time

template <int NP, int S, int U, int Q /* scalars per sample and step */, int NRED /* reduction buffers */>
struct Cfg {
  static constexpr int CL = NP / 128;
  static constexpr int E = S / 2;
  static constexpr int THREADS = 128 + 256 * U;
  static constexpr int KS = NP / 16;  // K steps
  // tensor memory columns: accumulators [unit][3][S] | three constant tiles of 8 | weights, NP/2 per matrix
  static constexpr int C_CONST = 3 * S * U;
  static constexpr int C_W = (C_CONST + 24 + 31) / 32 * 32;
  // K steps (of the 3*KS of the three matrices, in order) kept there; the rest in shared memory, tiles of four K steps
  static constexpr int NTK = NP == 512 ? (512 - C_W) / 32 * 4 : ((512 - C_W) / (NP / 2) > 3 ? 3 : (512 - C_W) / (NP / 2)) * KS;
  static constexpr int SM_TILES = (3 * KS - NTK) / 4;
  // shared memory
  static constexpr int ST_BUFS = CL > 1 ? 2 : 1;
  static constexpr int ST_ROW = NP == 512 ? 32 : 128;  // bytes of an operand row
  static constexpr int ST_BYTES = NP * ST_ROW;
  static constexpr int RED_BUFS = S < 64 && NP < 512 ? 2 : 1;  // alternating, so that one barrier per step is enough
  static constexpr int RED_BYTES = 128 * S * 4;
  static constexpr int OFF_W = U * ST_BUFS * ST_BYTES;
  static constexpr int OFF_RED = OFF_W + SM_TILES * 16384;
  static constexpr int OFF_SC = OFF_RED + U * NRED * RED_BUFS * RED_BYTES;
  static constexpr int SC_BYTES = 2 * CH * Q * S * 4;             // per unit
  static constexpr int OFF_DEC = OFF_SC + U * SC_BYTES;
  static constexpr int DEC_BYTES = Q == 2 ? 2 * 3 * S * 8 * 4 : 0;  // forward: eight steps of decode sums, twice
  static constexpr int OFF_UV = OFF_DEC + U * DEC_BYTES;
  static constexpr int OFF_BAR = OFF_UV + 128 * 8;
  static constexpr int SMEM = OFF_BAR + 256 + 1024;
  static_assert(SMEM <= tcr::SMEM_LIMIT, "shared memory");
  static_assert(NTK % 4 == 0 && NTK >= KS && C_W + NTK * 8 <= 512, "tensor memory");
  static_assert(NP < 512 || S == 16, "operand rows of 16 samples");
  // registers: launched with LAUNCH_REGS per thread; the four service warps hand theirs to the epilogue
  static constexpr int LAUNCH_REGS = 65536 / THREADS / 8 * 8;
  static constexpr int LOW = U == 1 ? 72 : 40, HIGH = U == 1 ? 208 : 104;
  static_assert((4 * LOW + 8 * U * HIGH) * 32 <= LAUNCH_REGS * THREADS, "setmaxnreg budget");
};

// barrier block
constexpr uint32_t B_STATE = 0;      // [units x CTAs of the cluster <= 4][2] that CTA's neurons of the next operand are complete:
                                     // the two are used alternately, because a CTA may send the state after the next before
                                     // a third one's arrival for this one lands
constexpr uint32_t B_DFULL = 64;     // [2] the accumulators of the step are complete
constexpr uint32_t B_SC_FULL = 80;   // [2 units][2]
constexpr uint32_t B_SC_FREE = 112;  // [2 units][2]
constexpr uint32_t B_TMEM = 144;
constexpr uint32_t B_DEAD = 148;

template <class C>
struct Ctx {
  uint32_t base, bars, tmem;
  uint8_t* gen;
  uint32_t rank;
  WaitCtx w;
};

template <class C>
__device__ __forceinline__ Ctx<C> setup(uint8_t* smem_raw, int units, const float* dec_u, const float* dec_v, int N,
                                        int* status, volatile int* host) {
  Ctx<C> c;
  c.base = (smem_u32(smem_raw) + 1023u) & ~1023u;
  c.gen = smem_raw + (c.base - smem_u32(smem_raw));
  c.bars = c.base + C::OFF_BAR;
  c.rank = C::CL > 1 ? cluster_ctarank() : 0u;
  volatile int* dead = reinterpret_cast<volatile int*>(c.gen + C::OFF_BAR + B_DEAD);
  c.w = WaitCtx{dead, status, WAIT_LIMIT_CYCLES, host};
  const int warp = threadIdx.x >> 5;
  if (threadIdx.x == 0) {
    *dead = 0;
    for (int u = 0; u < units; ++u) {
      mbar_init(c.bars + B_DFULL + 8 * u, 1);
      for (int i = 0; i < 2; ++i) {
        // own neurons: one arrival per epilogue warp; a peer's: counted in bytes, armed by the MMA warp
        for (int q = 0; q < C::CL; ++q)
          mbar_init(c.bars + B_STATE + 16 * (u * C::CL + q) + 8 * i, q == (int)c.rank ? 8 : 1);
        mbar_init(c.bars + B_SC_FULL + 16 * u + 8 * i, 1);
        mbar_init(c.bars + B_SC_FREE + 16 * u + 8 * i, 8);
      }
    }
    fence_mbar_init();
  }
  if (threadIdx.x < 128) {
    const int n = (int)c.rank * 128 + threadIdx.x;
    float2 uv = make_float2(0.f, 0.f);
    if (dec_u != nullptr && n < N) uv = make_float2(dec_u[n], dec_v[n]);
    reinterpret_cast<float2*>(c.gen + C::OFF_UV)[threadIdx.x] = uv;
  }
  if (warp == 1) tmem_alloc(c.bars + B_TMEM, 512);
  tcgen05_fence_before();
  __syncthreads();
  if (C::CL > 1) {  // every CTA's barriers exist before a peer signals them
    cluster_arrive();
    cluster_wait();
  }
  tcgen05_fence_after();
  c.tmem = *reinterpret_cast<volatile uint32_t*>(c.gen + C::OFF_BAR + B_TMEM);
  return c;
}

template <class C>
__device__ __forceinline__ void teardown(const Ctx<C>& c) {
  if (*c.w.dead) __nanosleep(200000);  // abandoned run: let MMAs in flight land before their accumulators are freed
  tcgen05_fence_before();
  __syncthreads();
  if (C::CL > 1) {
    cluster_arrive();
    cluster_wait();
  }
  if ((threadIdx.x >> 5) == 1) tmem_dealloc(c.tmem, 512);
}

// The A operand, by the eight epilogue warps of unit 0 (h = which half of the K range): matrix m as bf16, converted here
// from the caller's fp32 tensors.  Forward: row n of the operand is row n of W (a thread reads along its row, four columns
// at a time); reverse: column n of W (consecutive lanes read consecutive columns).
template <class C, int NP, bool TRANSPOSED>
__device__ __forceinline__ void load_weights(const Ctx<C>& c, const float* const* W, int N, bool vec, const float* cterm, int n,
                                             int row, int h, uint32_t lane_base) {
  for (int m = 0; m < 3; ++m) {
    const float* w = W[m];
    const bool live = w != nullptr && n < N;
#pragma unroll(NP < 512 ? 1 : 2)
    for (int k0 = h * (NP / 2); k0 < (h + 1) * (NP / 2); k0 += 16) {
      float v[16];
      if (TRANSPOSED) {
#pragma unroll
        for (int i = 0; i < 16; ++i) v[i] = (live && k0 + i < N) ? __ldg(w + (size_t)(k0 + i) * N + n) : 0.f;
      } else if (vec) {
#pragma unroll
        for (int i = 0; i < 16; i += 4) {
          float4 f = make_float4(0.f, 0.f, 0.f, 0.f);
          if (live && k0 + i < N) f = __ldg(reinterpret_cast<const float4*>(w + (size_t)n * N + k0 + i));
          v[i] = f.x; v[i + 1] = f.y; v[i + 2] = f.z; v[i + 3] = f.w;
        }
      } else {
#pragma unroll
        for (int i = 0; i < 16; ++i) v[i] = (live && k0 + i < N) ? __ldg(w + (size_t)n * N + k0 + i) : 0.f;
      }
      uint32_t pk[8];
#pragma unroll
      for (int i = 0; i < 8; ++i) pk[i] = pack_bf16x2(v[2 * i], v[2 * i + 1]);
      const int ks = m * C::KS + k0 / 16;
      if (ks < C::NTK) {
        tmem_st8(c.tmem + lane_base + C::C_W + ks * 8, pk);
      } else {
        const uint32_t tile = c.base + C::OFF_W + (ks - C::NTK) / 4 * 16384 + row * 128;
        const uint32_t u0 = (uint32_t)((ks - C::NTK) & 3) * 2;
#pragma unroll
        for (int i = 0; i < 2; ++i)
          asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(tile + (((u0 + i) ^ ((uint32_t)row & 7u)) << 4)),
                       "r"(pk[4 * i]), "r"(pk[4 * i + 1]), "r"(pk[4 * i + 2]), "r"(pk[4 * i + 3])
                       : "memory");
      }
    }
  }
  if (h == 0) {
    for (int i = 0; i < 3; ++i) {
      const uint32_t v = pack_bf16x2(cterm[i], cterm[i]);
      const uint32_t pk[8] = {v, v, v, v, v, v, v, v};
      tmem_st8(c.tmem + lane_base + C::C_CONST + 8 * i, pk);
    }
  }
  tmem_st_wait();
  if (C::SM_TILES > 0) fence_proxy_async_smem();
}

// MMA issuer (one whole warp, see umma_ts_warp; everything the instructions are built from is uniform).  Unit u's tile of
// a round exists iff tile + u * stride / U < n_ut.
template <class C, int NP, int S, int U>
__device__ __forceinline__ void mma_role(const Ctx<C>& c, int first, int stride, int n_ut, int T, int n_const, int code) {
  constexpr uint32_t idesc = make_idesc_bf16(128, S, 0, 1);
  const uint32_t lead = elect_one();
  const uint32_t tmem = __shfl_sync(0xffffffffu, c.tmem, 0), base = __shfl_sync(0xffffffffu, c.base, 0),
                 rank = __shfl_sync(0xffffffffu, c.rank, 0);
  uint32_t g[U];
#pragma unroll
  for (int u = 0; u < U; ++u) g[u] = 0;
  for (int tile = first; tile < n_ut; tile += stride) {
    for (int t = 0; t < T; ++t) {
#pragma unroll
      for (int u = 0; u < U; ++u) {
        if (tile + u * (stride / U) >= n_ut) continue;
        const uint32_t st = base + (u * C::ST_BUFS + (C::ST_BUFS > 1 ? (g[u] & 1u) : 0u)) * C::ST_BYTES;
        const uint32_t d = tmem + u * 3 * S;
        constexpr uint32_t B_STEP = C::ST_ROW;  // 16 rows, in units of 16 bytes
        // the neurons of one CTA at a time, this CTA's own first: the peers' are still on their way
        if (C::CL > 1 && lead) {
          for (uint32_t i = 1; i < C::CL; ++i)
            mbar_arrive_expect_tx(c.bars + B_STATE + 16 * (u * C::CL + (rank ^ i)) + 8 * (g[u] & 1u), 128 * S * 2);
        }
        __syncwarp();
#pragma unroll 1
        for (uint32_t i = 0; i < C::CL; ++i) {
          const uint32_t q = rank ^ i;
          const bool ok = mbar_wait<(C::CL > 1)>(c.bars + B_STATE + 16 * (u * C::CL + q) + 8 * (g[u] & 1u), (g[u] >> 1) & 1u, c.w, code);
          if (!__all_sync(0xffffffffu, ok)) return;
          if (C::CL > 1) fence_proxy_async_all();
          tcgen05_fence_after();
          const uint64_t b0 = (C::ST_ROW == 32 ? desc_sw32(desc_lo(st, 16)) : desc_sw128(desc_lo(st, 16))) + q * 8 * B_STEP;
#pragma unroll
          for (int m = 0; m < 3; ++m) {
#pragma unroll
            for (int ks = 0; ks < 8; ++ks) {
              const int w = m * C::KS + (int)q * 8 + ks;
              const bool acc = ks > 0 || i > 0;
              // where the K step is kept: known at compile time except for the one matrix that is cut (NP = 512)
              const bool in_tmem = (C::NTK % C::KS != 0 && m == C::NTK / C::KS) ? w < C::NTK : m < C::NTK / C::KS;
              if (in_tmem) {
                umma_ts_warp(d + m * S, tmem + C::C_W + w * 8, b0 + ks * B_STEP, idesc, acc, lead);
              } else {
                const uint64_t a0 = desc_sw128(desc_lo(base + C::OFF_W, 16));
                umma_ss_warp(d + m * S, a0 + (uint32_t)((w - C::NTK) / 4 * 1024 + 2 * ((w - C::NTK) & 3)), b0 + ks * B_STEP, idesc,
                             acc, lead);
              }
            }
          }
#pragma unroll 1
          for (int x = 0; x < n_const; ++x) {
#pragma unroll
            for (int ks = 0; ks < 8; ++ks)
              umma_ts_warp(d, tmem + C::C_CONST + 8 * x, b0 + ks * B_STEP, idesc, true, lead);
          }
        }
        if (lead) umma_commit(c.bars + B_DFULL + 8 * u);
        __syncwarp();
        ++g[u];
      }
    }
  }
}

// Publishes this thread's E new state values (packed bf16 pairs) into row `row` of operand buffer g & 1: sent to the peers
// (asynchronous stores, counted on their barriers), then stored here, where the MMAs on this CTA's own neurons start first.
// The reader of a peer's part orders it against the tensor core's reads by a proxy fence behind its wait.
template <class C, int S>
__device__ __forceinline__ void publish(const Ctx<C>& c, const uint32_t* packed, uint32_t g, int u, int row_k, int h,
                                        int lane) {
  const uint32_t parity = g & 1u;
  const uint32_t buf = c.base + (u * C::ST_BUFS + (C::ST_BUFS > 1 ? parity : 0u)) * C::ST_BYTES + row_k * C::ST_ROW;
  const uint32_t swizzle = C::ST_ROW == 32 ? ((uint32_t)row_k >> 2) & 1u : (uint32_t)row_k & 7u;
  const uint32_t bar = c.bars + B_STATE + 16 * (u * C::CL + c.rank) + 8 * parity;
  auto addr = [&](int v) { return buf + (((uint32_t)(h * (C::E / 8) + v) ^ swizzle) << 4); };
#pragma unroll
  for (uint32_t peer = 1; peer < C::CL; ++peer) {
    const uint32_t peer_bar = mapa(bar, c.rank ^ peer);
#pragma unroll
    for (int v = 0; v < C::E / 8; ++v)
      st_async_v4(mapa(addr(v), c.rank ^ peer), peer_bar, packed[4 * v], packed[4 * v + 1], packed[4 * v + 2], packed[4 * v + 3]);
  }
#pragma unroll
  for (int v = 0; v < C::E / 8; ++v)
    asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(addr(v)), "r"(packed[4 * v]), "r"(packed[4 * v + 1]),
                 "r"(packed[4 * v + 2]), "r"(packed[4 * v + 3])
                 : "memory");
  fence_proxy_async_smem();
  tcgen05_fence_before();  // this thread's accumulator reads precede the MMAs the arrival releases
  __syncwarp();
  if (lane == 0) mbar_arrive(bar);
}

// Scalar stage (one warp per unit): scalars of entry e = eight at a time, entry e of quantity i for sample s at
// sc[(e/8)&1][e%8][i][s].  src(i, b, e) reads quantity i of sample b (b < B) at entry e < T.
template <class C, int S, int Q, class Src>
__device__ __forceinline__ void scalar_role(const Ctx<C>& c, int u, int first, int stride, int n_ut, int T, int B, int code,
                                            Src src) {
  const int lane = threadIdx.x & 31;
  uint32_t chunk = 0;
  for (int tile = first; tile < n_ut; tile += stride) {
    const int b0 = tile * S;
    for (int e0 = 0; e0 < T; e0 += CH, ++chunk) {
      const uint32_t buf = chunk & 1u;
      if (chunk >= 2 && !mbar_wait(c.bars + B_SC_FREE + 16 * u + 8 * buf, ((chunk >> 1) - 1) & 1u, c.w, code)) return;
      float* sc = reinterpret_cast<float*>(c.gen + C::OFF_SC + u * C::SC_BYTES) + buf * (CH * Q * S);
#pragma unroll 1
      for (int i = 0; i < Q; ++i) {
#pragma unroll 4
        for (int x = lane; x < S * CH; x += 32) {
          const int s = x / CH, k = x % CH;
          const int b = b0 + s, e = e0 + k;
          sc[(k * Q + i) * S + s] = (b < B && e < T) ? src(i, b, e) : 0.f;
        }
      }
      __syncwarp();
      if (lane == 0) mbar_arrive(c.bars + B_SC_FULL + 16 * u + 8 * buf);
    }
  }
}

// 16-byte unit `unit` of neuron row n in a reduction buffer of [128 neurons][S samples] fp32: swizzled so that eight
// consecutive rows at the same unit fall into different banks
template <int S>
__device__ __forceinline__ uint32_t red_offset(int n, int unit) {
  const int sw = S == 16 ? ((n >> 1) & 3) : (n & 7);
  return (uint32_t)(n * S * 4 + ((unit ^ sw) << 4));
}

// Sum of NV values over the 16 lanes of a half warp, scattered: on return v[0..2] hold, for NV = 12, elements
// 6*bit3 + 3*bit2 + {0,1,2} of the lane (for NV = 8: v[0..1], elements 4*bit3 + 2*bit2 + {0,1}).  Fixed order.
template <int NV>
__device__ __forceinline__ void half_warp_sums(float* v, int lane) {
  static_assert(NV % 4 == 0, "two halvings");
#pragma unroll
  for (int i = 0; i < NV / 2; ++i) {
    const bool up = lane & 8;
    const float send = up ? v[i] : v[i + NV / 2], keep = up ? v[i + NV / 2] : v[i];
    v[i] = keep + __shfl_xor_sync(0xffffffffu, send, 8);
  }
#pragma unroll
  for (int i = 0; i < NV / 4; ++i) {
    const bool up = lane & 4;
    const float send = up ? v[i] : v[i + NV / 4], keep = up ? v[i + NV / 4] : v[i];
    v[i] = keep + __shfl_xor_sync(0xffffffffu, send, 4);
  }
#pragma unroll
  for (int i = 0; i < NV / 4; ++i) {
    v[i] += __shfl_xor_sync(0xffffffffu, v[i], 2);
    v[i] += __shfl_xor_sync(0xffffffffu, v[i], 1);
  }
}

__device__ __forceinline__ float4 lds4(const float* p) { return *reinterpret_cast<const float4*>(p); }

// private layouts of the saved tensors: piece v (8 samples) of a thread, 16 bytes per lane, 512 contiguous per warp
template <class C, int S>
__device__ __forceinline__ size_t dh_offset(int t, int n_ut, int ut, uint32_t rank, int h, int v, int row) {
  return ((((((size_t)t * n_ut + ut) * C::CL + rank) * 2 + h) * (C::E / 8) + v) * 128 + row) * 8;
}
// sign words: E <= 16: one word per thread (zero bits above the sign bits); E = 32: two
template <class C, int S>
__device__ __forceinline__ size_t sg_offset(int t, int n_ut, int ut, uint32_t rank, int h, int i, int row) {
  constexpr int WORDS = C::E > 16 ? 2 : 1;
  return (((((size_t)t * n_ut + ut) * C::CL + rank) * 2 + h) * WORDS + i) * 128 + row;
}

// One cluster per `units`-tile, never more than can be resident; what the launch needs from the driver is looked up once
// per kernel and device.
template <class C, class Launch>
int launch_lane(int slot, const void* kernel, int n_tiles, cudaStream_t s, Launch go) {
  cudaLaunchConfig_t cfg;
  memset(&cfg, 0, sizeof(cfg));
  cfg.blockDim = dim3(C::THREADS, 1, 1);
  cfg.dynamicSmemBytes = C::SMEM;
  cfg.stream = s;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = C::CL;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  const int resident = resident_clusters(kernel, &cfg, C::CL, C::SMEM);
  if (resident < 0) return RINGRNN_ERR_CUDA;
  cfg.gridDim = dim3((unsigned)((n_tiles < resident ? n_tiles : resident) * C::CL), 1, 1);
  {
    LaunchScope ls(slot, s);
    RINGRNN_CUDA_TRY(go(&cfg));
  }
  return RINGRNN_OK;
}

}  // namespace lane
}  // namespace ringrnn
