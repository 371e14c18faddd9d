// bf16 mode, forward, N <= 512: neurons on the tensor-memory lanes (see tc_lane.cuh for the decomposition).  One launch
// runs all T steps; the fp32 master state of S samples x 128 neurons lives in the registers of a unit's eight epilogue
// warps, S/2 values per thread.
#include <string.h>

#include "tc_lane.cuh"

namespace ringrnn {

using namespace lane;

template <int ACT, int NP, int S, int U>
__global__ void __launch_bounds__(128 + 256 * U, 1) fwd_lane_kernel(const __grid_constant__ LaneFwdParams p) {
  using C = Cfg<NP, S, U, 2, 1>;
  constexpr int E = C::E;
  extern __shared__ uint8_t smem_raw[];
  const Ctx<C> c = setup<C>(smem_raw, U, p.dec_u, p.dec_v, p.N, p.status, p.host);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int first = (int)(blockIdx.x / C::CL), groups = (int)(gridDim.x / C::CL), stride = groups * U;
  const int T = p.T;
  const bool epi = warp >= 4;
  const int u = epi ? (warp - 4) >> 3 : 0;            // unit
  const int h = ((warp - 4) >> 2) & 1, quarter = warp & 3;
  const int row = quarter * 32 + lane;                // lane of the accumulators = neuron within this CTA
  const int n = (int)c.rank * 128 + row;
  const uint32_t lane_base = (uint32_t)(quarter * 32) << 16;

  if (epi && u == 0) {
    const float* const W[3] = {p.use_wo ? p.Wo : nullptr, p.WL, p.WR};
    load_weights<C, NP, false>(c, W, p.N, p.w_vec != 0, p.cterm, n, row, h, lane_base);
  }
  tcgen05_fence_before();
  __syncthreads();
  tcgen05_fence_after();

  if (!epi) {
    tcr::reg_dec<C::LOW>();
    if (warp == 0) {
      mma_role<C, NP, S, U>(c, first, stride, p.n_ut, T, p.n_const, 202);
    } else if (warp >= 2 && warp - 2 < U) {
      scalar_role<C, S, 2>(c, warp - 2, first + (warp - 2) * groups, stride, p.n_ut, T, p.B, 203, [&](int i, int b, int e) {
        const int col = i == 0 ? p.colL : p.colR;
        return col >= 0 ? __ldg(p.A + ((size_t)b * p.T_total + p.t0 + e) * p.a_dim + col) : 0.f;
      });
    }
  } else {
    tcr::reg_inc<C::HIGH>();
    const bool live = n < p.N;
    const float J1 = live ? p.J1 : 0.f;  // padding neurons: the constant tile reaches them too, their state stays zero
    const f32x2 J1p = pk2(J1, J1), alphap = pk2(p.alpha, p.alpha), betap = pk2(1.f - p.alpha, 1.f - p.alpha);
    const bool want_ta = p.dec[0][2] != nullptr, want_dh = p.Dh != nullptr;
    const bool want_dec = p.dec[0][0] != nullptr || p.dec[0][1] != nullptr || p.dec[0][2] != nullptr;
    const int tid = threadIdx.x - 128 - 256 * u;  // within the unit
    const uint32_t d_base = c.tmem + lane_base + u * 3 * S + h * E;
    float* const red0 = reinterpret_cast<float*>(c.gen + C::OFF_RED + u * C::RED_BUFS * C::RED_BYTES);
    float* const decb = reinterpret_cast<float*>(c.gen + C::OFF_DEC + u * C::DEC_BYTES);
    const float2* const uv = reinterpret_cast<const float2*>(c.gen + C::OFF_UV);
    uint32_t g = 0, chunk = 0;
    for (int ut = first + u * groups; ut < p.n_ut; ut += stride) {
      const int b0 = ut * S + h * E;
      float master[E];
      uint32_t packed[E / 2];
#pragma unroll
      for (int j = 0; j < E; ++j) master[j] = (live && b0 + j < p.B) ? __ldg(p.r_init + (size_t)(b0 + j) * p.N + n) : 0.f;
#pragma unroll
      for (int j = 0; j < E / 2; ++j) packed[j] = pack_bf16x2(master[2 * j], master[2 * j + 1]);
      publish<C, S>(c, packed, g, u, n, h, lane);
      if (p.Rh != nullptr) {
        uint4* dst = reinterpret_cast<uint4*>(p.Rh + (size_t)n * p.BPs + b0);
#pragma unroll
        for (int v = 0; v < E / 8; ++v)
          dst[v] = make_uint4(packed[4 * v], packed[4 * v + 1], packed[4 * v + 2], packed[4 * v + 3]);
      }
      for (int t = 0; t < T; ++t, ++g) {
        const int k = t % CH;
        if (k == 0) mbar_wait(c.bars + B_SC_FULL + 16 * u + 8 * (chunk & 1u), (chunk >> 1) & 1u, c.w, 204);
        const float* sc = reinterpret_cast<const float*>(c.gen + C::OFF_SC + u * C::SC_BYTES) +
                          ((chunk & 1u) * CH + k) * (2 * S) + h * E;
        uint32_t dpk[E / 2], neg = 0u;
        float min_mag = 3.0e38f;
        mbar_wait(c.bars + B_DFULL + 8 * u, g & 1u, c.w, 205);
        tcgen05_fence_after();
        constexpr int GR = E < 16 ? E : 16;
#pragma unroll
        for (int j0 = 0; j0 < E; j0 += GR) {
          uint32_t yo[GR], yl[GR], yr[GR];
          if constexpr (GR == 8) {
            tmem_ld8(d_base, yo);
            tmem_ld8(d_base + S, yl);
            tmem_ld8(d_base + 2 * S, yr);
          } else {
            tmem_ld16(d_base + j0, yo);
            tmem_ld16(d_base + S + j0, yl);
            tmem_ld16(d_base + 2 * S + j0, yr);
          }
          tmem_ld_wait();
#pragma unroll
          for (int j1 = 0; j1 < GR; j1 += 8) {
            const float4 La = lds4(sc + j0 + j1), Lb = lds4(sc + j0 + j1 + 4);
            const float4 Ra = lds4(sc + S + j0 + j1), Rb = lds4(sc + S + j0 + j1 + 4);
            const f32x2 L2[4] = {pk2(La.x, La.y), pk2(La.z, La.w), pk2(Lb.x, Lb.y), pk2(Lb.z, Lb.w)};
            const f32x2 R2[4] = {pk2(Ra.x, Ra.y), pk2(Ra.z, Ra.w), pk2(Rb.x, Rb.y), pk2(Rb.z, Rb.w)};
            f32x2 re2[4], f2[4], d2[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) {
              const int e = j1 + 2 * i;
              f32x2 v = mul2(J1p, pk2u(yo[e], yo[e + 1]));
              v = fma2(L2[i], pk2u(yl[e], yl[e + 1]), v);
              re2[i] = fma2(R2[i], pk2u(yr[e], yr[e + 1]), v);
            }
            tcr::act_group2<ACT, 8>(re2, f2, d2);
#pragma unroll
            for (int i = 0; i < 4; ++i) {
              const int e = j0 + j1 + 2 * i;
              const f32x2 r2 = fma2(alphap, f2[i], mul2(betap, pk2(master[e], master[e + 1])));
              upk2(r2, master[e], master[e + 1]);
              packed[e / 2] = pack_bf16x2(master[e], master[e + 1]);
              if (want_dh) {
                float da, db;
                upk2(d2[i], da, db);
                dpk[e / 2] = pack_bf16x2(da, db);
              }
            }
          }
        }
        if (t + 1 < T) publish<C, S>(c, packed, g + 1, u, n, h, lane);
        // ---- off the critical path: the next step's MMAs are running
        if (k == CH - 1 || t + 1 == T) {  // the scalars of this chunk are no longer needed
          __syncwarp();
          if (lane == 0) mbar_arrive(c.bars + B_SC_FREE + 16 * u + 8 * (chunk & 1u));
          ++chunk;
        }
        if (want_dh) {
#pragma unroll
          for (int v = 0; v < E / 8; ++v)
            st_cs_v4(p.Dh + dh_offset<C, S>(t, p.n_ut, ut, c.rank, h, v, row), dpk[4 * v], dpk[4 * v + 1], dpk[4 * v + 2],
                     dpk[4 * v + 3]);
          // bits of the backward's d|r|/dr: sign bits (sample j at bit j), exact zeros (rare) above them
#pragma unroll
          for (int j = E - 1; j >= 0; --j) {
            neg = __funnelshift_l(__float_as_uint(master[j]), neg, 1);
            min_mag = fminf(min_mag, fabsf(master[j]));
          }
          uint32_t zero = 0u;
          if (min_mag == 0.f) {
#pragma unroll
            for (int j = 0; j < E; ++j) zero |= (master[j] == 0.f ? 1u : 0u) << j;
          }
          uint32_t* sg = p.Sg + sg_offset<C, S>(t, p.n_ut, ut, c.rank, h, 0, row);
          if constexpr (E > 16) {
            sg[0] = neg;
            sg[128] = zero;
          } else {
            sg[0] = neg | (zero << 16);
          }
          if (t + 1 < T) {
            uint4* dst = reinterpret_cast<uint4*>(p.Rh + ((size_t)(t + 1) * NP + n) * p.BPs + b0);
#pragma unroll
            for (int v = 0; v < E / 8; ++v)
              dst[v] = make_uint4(packed[4 * v], packed[4 * v + 1], packed[4 * v + 2], packed[4 * v + 3]);
          }
        }
        if (p.ckpt != nullptr && live && t + 1 < T && (t + 1) % p.ckpt_every == 0) {
          float* dst = p.ckpt + ((size_t)((t + 1) / p.ckpt_every) * p.B + b0) * p.N + n;
#pragma unroll
          for (int j = 0; j < E; ++j)
            if (b0 + j < p.B) dst[(size_t)j * p.N] = master[j];
        }
        if (p.hist != nullptr && live) {
          float* dst = p.hist + ((size_t)t * p.B + b0) * p.N + n;
#pragma unroll
          for (int j = 0; j < E; ++j)
            if (b0 + j < p.B) dst[(size_t)j * p.N] = master[j];
        }
        if (want_dec) {
          // x = r.u, y = r.v, sum|r| over this CTA's neurons: the fp32 state through shared memory, then S/4 x 16 threads
          // (four samples, every 16th neuron each) and a fixed-order reduction over the 16
          float* red = red0 + (C::RED_BUFS > 1 ? (t & 1) : 0) * (C::RED_BYTES / 4);
          if (C::RED_BUFS == 1) named_bar_sync(4 + u, 256);  // the previous step's readers are done
#pragma unroll
          for (int v = 0; v < E / 4; ++v)
            *reinterpret_cast<float4*>(reinterpret_cast<uint8_t*>(red) + red_offset<S>(row, h * (E / 4) + v)) =
                make_float4(master[4 * v], master[4 * v + 1], master[4 * v + 2], master[4 * v + 3]);
          named_bar_sync(2 + u, 256);
          float* dec_t = decb + ((t / 8) & 1) * (3 * S * 8);
          if (tid < 4 * S) {
            const int part = tid & 15, quad = tid >> 4;
            float a[12];
#pragma unroll
            for (int i = 0; i < 12; ++i) a[i] = 0.f;
#pragma unroll
            for (int i = 0; i < 8; ++i) {
              const int nn = part + 16 * i;
              const float4 r = lds4(reinterpret_cast<const float*>(reinterpret_cast<const uint8_t*>(red) + red_offset<S>(nn, quad)));
              const float2 w = uv[nn];
              a[0] = fmaf(r.x, w.x, a[0]); a[1] = fmaf(r.y, w.x, a[1]); a[2] = fmaf(r.z, w.x, a[2]); a[3] = fmaf(r.w, w.x, a[3]);
              a[4] = fmaf(r.x, w.y, a[4]); a[5] = fmaf(r.y, w.y, a[5]); a[6] = fmaf(r.z, w.y, a[6]); a[7] = fmaf(r.w, w.y, a[7]);
              if (want_ta) {
                a[8] += fabsf(r.x); a[9] += fabsf(r.y); a[10] += fabsf(r.z); a[11] += fabsf(r.w);
              }
            }
            auto put = [&](int v0, int n) {  // the first n of a[] are values v0.. of [kind][sample of the quad]
#pragma unroll
              for (int i = 0; i < 3; ++i)
                if (i < n) dec_t[((v0 + i) / 4 * S + quad * 4 + (v0 + i) % 4) * 8 + (t & 7)] = a[i];
            };
            if (want_ta) {
              half_warp_sums<12>(a, lane);
              if ((lane & 3) == 0) put(6 * ((lane >> 3) & 1) + 3 * ((lane >> 2) & 1), 3);
            } else {  // a roll-out asks for the two angles' sums only
              half_warp_sums<8>(a, lane);
              if ((lane & 3) == 0) put(4 * ((lane >> 3) & 1) + 2 * ((lane >> 2) & 1), 2);
            }
          }
          // eight steps at a time to global memory, one chunk behind: the barrier above orders the sums of the
          // previous chunk before this read of them, and nobody writes that chunk's buffer again for eight steps
          if ((t & 7) == 0 && t > 0) {
            const float* src = decb + (((t / 8) & 1) ^ 1) * (3 * S * 8);
            for (int i = tid; i < 3 * S; i += 256) {
              const int kind = i / S, b = ut * S + i % S;
              float* o = p.dec[c.rank][kind];
              if (b < p.B && o != nullptr) {
                o += (size_t)b * T + (t - 8);
                const float4 x = lds4(src + i * 8), y = lds4(src + i * 8 + 4);
                if (p.dec_vec) {
                  reinterpret_cast<float4*>(o)[0] = x;
                  reinterpret_cast<float4*>(o)[1] = y;
                } else {
                  o[0] = x.x; o[1] = x.y; o[2] = x.z; o[3] = x.w; o[4] = y.x; o[5] = y.y; o[6] = y.z; o[7] = y.w;
                }
              }
            }
          }
        }
      }
      if (want_dec) {  // the last (up to eight) steps of the tile
        named_bar_sync(2 + u, 256);
        const int t1 = (T - 1) / 8 * 8;
        const float* src = decb + ((t1 / 8) & 1) * (3 * S * 8);
        for (int i = tid; i < 3 * S; i += 256) {
          const int kind = i / S, b = ut * S + i % S;
          float* o = p.dec[c.rank][kind];
          if (b < p.B && o != nullptr) {
            o += (size_t)b * T + t1;
            for (int x = 0; x < T - t1; ++x) o[x] = src[i * 8 + x];
          }
        }
        named_bar_sync(2 + u, 256);  // read before the next tile's first sums
      }
      if (p.final_state != nullptr && live) {
#pragma unroll
        for (int j = 0; j < E; ++j)
          if (b0 + j < p.B) p.final_state[(size_t)(b0 + j) * p.N + n] = master[j];
      }
    }
  }
  teardown<C>(c);
}

namespace {

template <int ACT, int NP, int S, int U>
int launch(const LaneFwdParams& p, cudaStream_t s) {
  using C = Cfg<NP, S, U, 2, 1>;
  auto kernel = fwd_lane_kernel<ACT, NP, S, U>;
  return launch_lane<C>(K_FWD, reinterpret_cast<const void*>(kernel), (p.n_ut + U - 1) / U, s,
                        [&](const cudaLaunchConfig_t* cfg) { return cudaLaunchKernelEx(cfg, kernel, p); });
}

template <int ACT>
int by_shape(int NP, int S, int U, const LaneFwdParams& p, cudaStream_t s) {
  if (NP == 128) {
    if (U == 2) return launch<ACT, 128, 64, 2>(p, s);
    if (S == 16) return launch<ACT, 128, 16, 1>(p, s);
    if (S == 32) return launch<ACT, 128, 32, 1>(p, s);
    return launch<ACT, 128, 64, 1>(p, s);
  }
  if (NP == 512) return launch<ACT, 512, 16, 1>(p, s);
  if (S == 16) return launch<ACT, 256, 16, 1>(p, s);
  if (S == 32) return launch<ACT, 256, 32, 1>(p, s);
  return launch<ACT, 256, 64, 1>(p, s);
}

}  // namespace

int lane_forward_launch(int act, int NP, int S, int units, const LaneFwdParams& p, cudaStream_t s) {
  switch (act) {
    case RINGRNN_ACT_RELU: return by_shape<RINGRNN_ACT_RELU>(NP, S, units, p, s);
    case RINGRNN_ACT_GELU: return by_shape<RINGRNN_ACT_GELU>(NP, S, units, p, s);
    case RINGRNN_ACT_SILU: return by_shape<RINGRNN_ACT_SILU>(NP, S, units, p, s);
    default: return by_shape<RINGRNN_ACT_TANH>(NP, S, units, p, s);
  }
}

}  // namespace ringrnn
