// bf16 mode, reverse time, N <= 512: neurons on the tensor-memory lanes (see tc_lane.cuh for the decomposition).  Per step
//   D_m[j, sample] = W_m^T x delta_t      carry = (1-alpha) g + J0 sum_i delta + J1 Zo + L Zl + R Zr
//   g_{t-1} = carry + dL/dr_{t-1}         delta_{t-1} = alpha F'(re_{t-1}) g_{t-1}
// delta, L*delta and R*delta go to DL, [T][3][NP][samples], the K-major A operand of the weight-gradient GEMM.
#include <string.h>

#include "tc_lane.cuh"

namespace ringrnn {

using namespace lane;

template <int NP, int S>
__global__ void __launch_bounds__(384, 1) bwd_lane_kernel(const __grid_constant__ LaneBwdParams p) {
  using C = Cfg<NP, S, 1, 5, NP < 512 ? 2 : 1>;
  constexpr int E = C::E;
  constexpr int NRED = NP < 512 ? 2 : 1;  // dL/dA: both products side by side, or one after the other
  extern __shared__ uint8_t smem_raw[];
  const Ctx<C> c = setup<C>(smem_raw, 1, p.dec_u, p.dec_v, p.N, p.status, p.host);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int first = (int)(blockIdx.x / C::CL), stride = (int)(gridDim.x / C::CL);
  const int T = p.T;
  const bool epi = warp >= 4;
  const int h = ((warp - 4) >> 2) & 1, quarter = warp & 3;
  const int row = quarter * 32 + lane;
  const int n = (int)c.rank * 128 + row;
  const uint32_t lane_base = (uint32_t)(quarter * 32) << 16;

  if (epi) {
    const float* const W[3] = {p.use_wo ? p.Wo : nullptr, p.WL, p.WR};
    load_weights<C, NP, true>(c, W, p.N, false, p.cterm, n, row, h, lane_base);
  }
  tcgen05_fence_before();
  __syncthreads();
  tcgen05_fence_after();

  if (!epi) {
    tcr::reg_dec<C::LOW>();
    if (warp == 0) {
      mma_role<C, NP, S, 1>(c, first, stride, p.n_ut, T, p.n_const, 302);
    } else if (warp == 2) {
      // entry e belongs to step T-1-e: L, R, coef_x, coef_y, coef_s
      scalar_role<C, S, 5>(c, 0, first, stride, p.n_ut, T, p.B, 303, [&](int i, int b, int e) {
        const size_t bt = (size_t)b * p.T_total + p.t0 + (T - 1 - e);
        if (i < 2) {
          const int col = i == 0 ? p.colL : p.colR;
          return col >= 0 ? __ldg(p.A + bt * p.a_dim + col) : 0.f;
        }
        const float* src = i == 2 ? p.coef_x : i == 3 ? p.coef_y : p.coef_s;
        return src != nullptr ? __ldg(src + bt) : 0.f;
      });
    }
  } else {
    tcr::reg_inc<C::HIGH>();
    const bool live = n < p.N;
    const float J1 = live ? p.J1 : 0.f;  // the constant tile reaches padding neurons too; their delta stays zero
    const f32x2 J1p = pk2(J1, J1), betap = pk2(1.f - p.alpha, 1.f - p.alpha), alphap = pk2(p.alpha, p.alpha);
    const bool has_coef = p.coef_x != nullptr, want_dA = p.dA_part != nullptr;
    const int tid = threadIdx.x - 128;
    const uint32_t d_base = c.tmem + lane_base + h * E;
    const float2 uvn = reinterpret_cast<const float2*>(c.gen + C::OFF_UV)[row];
    const f32x2 un = pk2(uvn.x, uvn.x), vn = pk2(uvn.y, uvn.y);
    const float* const sc0 = reinterpret_cast<const float*>(c.gen + C::OFF_SC) + h * E;
    // scalar i of entry e, first of this thread's samples; `ch` = running number of the entry's chunk
    auto scal = [&](uint32_t ch, int e, int i) { return sc0 + (((ch & 1u) * CH + (e % CH)) * 5 + i) * S; };
    uint32_t g = 0, chunk0 = 0;  // chunk0: chunks consumed by earlier tiles
    for (int ut = first; ut < p.n_ut; ut += stride) {
      const int b0 = ut * S + h * E;
      float master[E];  // carry, then g_t
      uint4 dv[E / 8];  // F'(re) of the step about to be produced
      uint32_t neg = 0u, zero = 0u;
      float go[E];      // its part of dL/dr from grad_output
      auto prefetch = [&](int t) {
#pragma unroll
        for (int v = 0; v < E / 8; ++v) dv[v] = ld_cs_v4(p.Dh + dh_offset<C, S>(t, p.n_ut, ut, c.rank, h, v, row));
        if (has_coef) {
          const uint32_t* sg = p.Sg + sg_offset<C, S>(t, p.n_ut, ut, c.rank, h, 0, row);
          if constexpr (E > 16) {
            neg = __ldg(sg);
            zero = __ldg(sg + 128);
          } else {
            const uint32_t w = __ldg(sg);
            neg = w & 0xffffu;
            zero = w >> 16;
          }
        }
        if (p.grad_output != nullptr) {
          const float* src = p.grad_output + ((size_t)(p.t0 + t) * p.B + b0) * p.N + n;
#pragma unroll
          for (int j = 0; j < E; ++j) go[j] = (live && b0 + j < p.B) ? __ldg(src + (size_t)j * p.N) : 0.f;
        }
      };
      uint32_t packed[E / 2];
      // g_t from the carry, delta_t from g_t, entry e = T-1-t: into the operand buffer and DL
      auto produce = [&](int t, int e) {
        const uint32_t ch = chunk0 + (uint32_t)(e / CH);
        if (p.grad_output != nullptr) {
#pragma unroll
          for (int j = 0; j < E; ++j) master[j] += go[j];
        }
        if (has_coef && zero != 0u) {  // sign(0) = 0: taken out beforehand (rare)
          const float* cs = scal(ch, e, 4);
#pragma unroll
          for (int j = 0; j < E; ++j)
            if (zero & (1u << j)) master[j] -= (neg & (1u << j)) ? -cs[j] : cs[j];
        }
#pragma unroll
        for (int j = 0; j < E; j += 4) {
          f32x2 ga = pk2(master[j], master[j + 1]), gb = pk2(master[j + 2], master[j + 3]);
          if (has_coef) {
            const float4 cx = lds4(scal(ch, e, 2) + j), cy = lds4(scal(ch, e, 3) + j), cs = lds4(scal(ch, e, 4) + j);
            ga = fma2(pk2(cx.x, cx.y), un, ga);
            gb = fma2(pk2(cx.z, cx.w), un, gb);
            ga = fma2(pk2(cy.x, cy.y), vn, ga);
            gb = fma2(pk2(cy.z, cy.w), vn, gb);
            // + cs * sign(r) by the sign bit
            const f32x2 one = pk2(1.f, 1.f);
            ga = fma2(one, pk2((neg & (1u << j)) ? -cs.x : cs.x, (neg & (2u << j)) ? -cs.y : cs.y), ga);
            gb = fma2(one, pk2((neg & (4u << j)) ? -cs.z : cs.z, (neg & (8u << j)) ? -cs.w : cs.w), gb);
          }
          upk2(ga, master[j], master[j + 1]);
          upk2(gb, master[j + 2], master[j + 3]);
          const uint4 d4 = dv[j / 8];
          const uint32_t w0 = (j & 4) ? d4.z : d4.x, w1 = (j & 4) ? d4.w : d4.y;
          float x0, x1, x2, x3;
          upk2(mul2(mul2(alphap, pk2(tcr::bf16_lo(w0), tcr::bf16_hi(w0))), ga), x0, x1);
          upk2(mul2(mul2(alphap, pk2(tcr::bf16_lo(w1), tcr::bf16_hi(w1))), gb), x2, x3);
          packed[j / 2] = pack_bf16x2(x0, x1);
          packed[j / 2 + 1] = pack_bf16x2(x2, x3);
        }
        publish<C, S>(c, packed, g, 0, n, h, lane);
      };
      // off the critical path: delta_t and its scaled copies (packed bf16 products, the scalars rounded to bf16)
      auto write_dl = [&](int t, int e) {
        const uint32_t ch = chunk0 + (uint32_t)(e / CH);
        uint4* dst = reinterpret_cast<uint4*>(p.DL + ((size_t)t * 3 * NP + n) * p.BPs + b0);
        const size_t step = (size_t)NP * p.BPs / 8;
#pragma unroll
        for (int v = 0; v < E / 8; ++v) {
          dst[v] = make_uint4(packed[4 * v], packed[4 * v + 1], packed[4 * v + 2], packed[4 * v + 3]);
#pragma unroll
          for (int m = 0; m < 2; ++m) {
            const float4 a = lds4(scal(ch, e, m) + 8 * v), b = lds4(scal(ch, e, m) + 8 * v + 4);
            dst[(1 + m) * step + v] = make_uint4(tcr::mul_bf16x2(packed[4 * v], pack_bf16x2(a.x, a.y)),
                                                 tcr::mul_bf16x2(packed[4 * v + 1], pack_bf16x2(a.z, a.w)),
                                                 tcr::mul_bf16x2(packed[4 * v + 2], pack_bf16x2(b.x, b.y)),
                                                 tcr::mul_bf16x2(packed[4 * v + 3], pack_bf16x2(b.z, b.w)));
          }
        }
      };
      auto wait_entry = [&](int e) {  // the first entry of a chunk: its scalars are in shared memory
        if (e % CH == 0) {
          const uint32_t ch = chunk0 + (uint32_t)(e / CH);
          mbar_wait(c.bars + B_SC_FULL + 8 * (ch & 1u), (ch >> 1) & 1u, c.w, 304);
        }
      };

#pragma unroll
      for (int j = 0; j < E; ++j)
        master[j] = (p.carry_in != nullptr && live && b0 + j < p.B) ? __ldg(p.carry_in + (size_t)(b0 + j) * p.N + n) : 0.f;
      prefetch(T - 1);
      wait_entry(0);
      produce(T - 1, 0);
      write_dl(T - 1, 0);
      if (T > 1) prefetch(T - 2);
      for (int t = T - 1; t >= 0; --t, ++g) {
        const int e = T - 1 - t;
        const uint32_t ch = chunk0 + (uint32_t)(e / CH);
        uint4 rp[E / 8];  // r_{t-1} (bf16), for dL/dA
        if (want_dA) {
          const uint4* src = reinterpret_cast<const uint4*>(p.Rh + ((size_t)t * NP + n) * p.BPs + b0);
#pragma unroll
          for (int v = 0; v < E / 8; ++v) rp[v] = __ldg(src + v);
        }
        if (t > 0) wait_entry(e + 1);
        mbar_wait(c.bars + B_DFULL, g & 1u, c.w, 305);
        tcgen05_fence_after();
        float* red = reinterpret_cast<float*>(c.gen + C::OFF_RED) + (C::RED_BUFS > 1 ? (t & 1) : 0) * (NRED * C::RED_BYTES / 4);
        if (want_dA && C::RED_BUFS == 1) named_bar_sync(4, 256);  // the previous step's readers are done
        float later[NRED == 1 ? E : 4];
        constexpr int GR = E < 16 ? E : 16;
#pragma unroll
        for (int j0 = 0; j0 < E; j0 += GR) {
          uint32_t zo[GR], zl[GR], zr[GR];
          if constexpr (GR == 8) {
            tmem_ld8(d_base, zo);
            tmem_ld8(d_base + S, zl);
            tmem_ld8(d_base + 2 * S, zr);
          } else {
            tmem_ld16(d_base + j0, zo);
            tmem_ld16(d_base + S + j0, zl);
            tmem_ld16(d_base + 2 * S + j0, zr);
          }
          tmem_ld_wait();
#pragma unroll
          for (int j1 = 0; j1 < GR; j1 += 4) {
            const float4 L = lds4(scal(ch, e, 0) + j0 + j1), R = lds4(scal(ch, e, 1) + j0 + j1);
            const f32x2 L2[2] = {pk2(L.x, L.y), pk2(L.z, L.w)}, R2[2] = {pk2(R.x, R.y), pk2(R.z, R.w)};
#pragma unroll
            for (int i = 0; i < 2; ++i) {
              const int x = j1 + 2 * i, idx = j0 + x;
              f32x2 cv = mul2(betap, pk2(master[idx], master[idx + 1]));
              cv = fma2(J1p, pk2u(zo[x], zo[x + 1]), cv);
              cv = fma2(L2[i], pk2u(zl[x], zl[x + 1]), cv);
              cv = fma2(R2[i], pk2u(zr[x], zr[x + 1]), cv);
              upk2(cv, master[idx], master[idx + 1]);
            }
          }
          if (want_dA) {
            // products r_{t-1} * Zl, r_{t-1} * Zr of this neuron, to be summed over the neurons below
#pragma unroll
            for (int x = 0; x < GR; x += 4) {
              const uint4 r8 = rp[(j0 + x) / 8];
              const uint32_t w0 = (x & 4) ? r8.z : r8.x, w1 = (x & 4) ? r8.w : r8.y;
              const float r0 = tcr::bf16_lo(w0), r1 = tcr::bf16_hi(w0), r2 = tcr::bf16_lo(w1), r3 = tcr::bf16_hi(w1);
              if constexpr (NRED == 1) {  // the second product waits in registers
                later[j0 + x] = r0 * __uint_as_float(zr[x]);
                later[j0 + x + 1] = r1 * __uint_as_float(zr[x + 1]);
                later[j0 + x + 2] = r2 * __uint_as_float(zr[x + 2]);
                later[j0 + x + 3] = r3 * __uint_as_float(zr[x + 3]);
              }
              uint8_t* dst = reinterpret_cast<uint8_t*>(red) + red_offset<S>(row, (h * E + j0 + x) / 4);
              *reinterpret_cast<float4*>(dst) = make_float4(r0 * __uint_as_float(zl[x]), r1 * __uint_as_float(zl[x + 1]),
                                                            r2 * __uint_as_float(zl[x + 2]), r3 * __uint_as_float(zl[x + 3]));
              if constexpr (NRED == 2)
                *reinterpret_cast<float4*>(dst + C::RED_BYTES) = make_float4(r0 * __uint_as_float(zr[x]), r1 * __uint_as_float(zr[x + 1]), r2 * __uint_as_float(zr[x + 2]),
                              r3 * __uint_as_float(zr[x + 3]));
            }
          }
        }
        if (t > 0) {
          // (the operand buffers alternate with the step they serve: g counts it)
          ++g;
          produce(t - 1, e + 1);
          --g;
          write_dl(t - 1, e + 1);
        } else if (p.grad_r_init != nullptr && live) {
#pragma unroll
          for (int j = 0; j < E; ++j)
            if (b0 + j < p.B) p.grad_r_init[(size_t)(b0 + j) * p.N + n] = master[j];
        }
        if (e % CH == CH - 1 || t == 0) {  // nothing reads this chunk's scalars any more
          __syncwarp();
          if (lane == 0) mbar_arrive(c.bars + B_SC_FREE + 8 * (ch & 1u));
        }
        if (t > 1) prefetch(t - 2);
        if (want_dA) {
          const int part = tid & 15, quad = tid >> 4;
#pragma unroll
          for (int pass = 0; pass < 3 - NRED; ++pass) {
            if constexpr (NRED == 1) {
              if (pass == 1) {
                named_bar_sync(4, 256);  // the first product's readers are done
#pragma unroll
                for (int x = 0; x < E; x += 4)
                  *reinterpret_cast<float4*>(reinterpret_cast<uint8_t*>(red) + red_offset<S>(row, (h * E + x) / 4)) =
                      make_float4(later[x], later[x + 1], later[x + 2], later[x + 3]);
              }
            }
            named_bar_sync(2, 256);
            if (tid < 4 * S) {
              float a[4 * NRED];
#pragma unroll
              for (int i = 0; i < 4 * NRED; ++i) a[i] = 0.f;
#pragma unroll
              for (int i = 0; i < 8; ++i)
#pragma unroll
                for (int k = 0; k < NRED; ++k) {
                  const float4 v = lds4(reinterpret_cast<const float*>(reinterpret_cast<const uint8_t*>(red) + k * C::RED_BYTES +
                                                                       red_offset<S>(part + 16 * i, quad)));
                  a[4 * k] += v.x; a[4 * k + 1] += v.y; a[4 * k + 2] += v.z; a[4 * k + 3] += v.w;
                }
              half_warp_sums<4 * NRED>(a, lane);
              if ((lane & 3) == 0) {
                const int v0 = NRED * (2 * ((lane >> 3) & 1) + ((lane >> 2) & 1));
#pragma unroll
                for (int i = 0; i < NRED; ++i) {
                  const int k = NRED == 2 ? (v0 + i) / 4 : pass;
                  p.dA_part[(((size_t)c.rank * 2 + k) * T + t) * p.BPs + ut * S + quad * 4 + (v0 + i) % 4] = a[i];
                }
              }
            }
          }
        }
      }
      chunk0 += (uint32_t)((T + CH - 1) / CH);
    }
  }
  teardown<C>(c);
}

namespace {

template <int NP, int S>
int launch(const LaneBwdParams& p, cudaStream_t s) {
  using C = Cfg<NP, S, 1, 5, NP < 512 ? 2 : 1>;
  auto kernel = bwd_lane_kernel<NP, S>;
  return launch_lane<C>(K_BWD, reinterpret_cast<const void*>(kernel), p.n_ut, s,
                        [&](const cudaLaunchConfig_t* cfg) { return cudaLaunchKernelEx(cfg, kernel, p); });
}

}  // namespace

int lane_backward_launch(int NP, int S, const LaneBwdParams& p, cudaStream_t s) {
  if (NP == 128) return S == 16 ? launch<128, 16>(p, s) : S == 32 ? launch<128, 32>(p, s) : launch<128, 64>(p, s);
  if (NP == 512) return launch<512, 16>(p, s);
  return S == 16 ? launch<256, 16>(p, s) : S == 32 ? launch<256, 32>(p, s) : launch<256, 64>(p, s);
}

}  // namespace ringrnn
