// The x pass of the FLC scan over axes of any length (see genpass_dev.cuh).
#include "genpass_dev.cuh"

namespace tmb {

namespace {

// FLC: the rotated mask's spectrum times the spectra of f and f^2 (statistics, always
// complex64) and the template's times the spectrum of f; three tiles, one set of barriers.
template <int W, typename HT>
__global__ void __launch_bounds__(kMaxThreads, 1)
gen_xpass_flc_kernel(const float2* __restrict__ Gt, const float2* __restrict__ Gm,
                     const float2* __restrict__ Ft, const float2* __restrict__ Ft2, int B,
                     int per, int t0, int n1, int h2, const Plan p,
                     const float4* __restrict__ tw_g, float scale, HT* __restrict__ Ht,
                     float2* __restrict__ Hm, float2* __restrict__ Hm2, const HLayout hl) {
  extern __shared__ float4 smem_raw[];
  const int w = lines<W>(p), tid = threadIdx.x, nt = blockDim.x, l = tid % w, slot = tid / w;
  float4* tw = smem_raw;
  float2* sm = reinterpret_cast<float2*>(tw + p.pairs);
  const int tile = p.rows * w;  // tiles: mask (then CC(f, m)), template, CC(f^2, m)
  const int k2 = blockIdx.x * w + l, k1 = blockIdx.y;
  const bool valid = k2 < h2;  // the row padding is transformed as zeros
  for (int i = tid; i < p.pairs; i += nt) tw[i] = tw_g[i];
  __syncthreads();
  const int64_t row_s = (int64_t)n1 * h2, col = (int64_t)k1 * h2 + min(k2, h2 - 1);
  const int64_t in_step = p.lr[0] * row_s, out_step = p.lr[0] * hl.sx;
  auto input = [&](const float2* a) {  // the scale of H goes in with the few inputs
    return [=](int r) {
      if (!valid) return make_float2(0.f, 0.f);
      const float2 c = __ldg(a + r * in_step);
      return make_float2(c.x * scale, c.y * scale);
    };
  };
  auto output = [&](auto* a) {
    return [=](int r, float2 v) { store_c(a + r * out_step, v); };
  };
  const int b1 = min(B, (int)(blockIdx.z + 1) * per);
  for (int b = blockIdx.z * per; b < b1; ++b) {
    const int64_t g0 = (int64_t)b * t0 * row_s + col;
    TM_RADIX(p.r[0], ({
      first_stage<W, RR, -1, true>(p, sm, tw, l, slot, t0,
                                   [&](int q) { return input(Gm + g0 + q * row_s); });
      first_stage<W, RR, -1, true>(p, sm + tile, tw, l, slot, t0,
                                   [&](int q) { return input(Gt + g0 + q * row_s); });
    }));
    __syncthreads();
    for (int s = 1; s < p.ns - 1; ++s) {
      TM_RADIX(p.r[s], ({
        mid_stage<W, RR, -1>(p, s, sm, tw, l, slot);
        mid_stage<W, RR, -1>(p, s, sm + tile, tw, l, slot);
      }));
      __syncthreads();
    }
    TM_RADIX(p.rl, ({
      const int64_t step = (p.n / RR) * row_s;
      last_stage<W, RR, -1>(p, sm, l, slot, [&](int q, float2(&v)[RR], float2* d) {
        const int64_t at = col + out_base(p, q) * row_s;
        float2 u[RR];
        _Pragma("unroll")
        for (int r = 0; r < RR; ++r) u[r] = fft::cmul(v[r], __ldg(Ft2 + at + r * step));
        fft::dft_small<RR, 1>(u);
        _Pragma("unroll")
        for (int r = 0; r < RR; ++r) d[2 * tile + r * w] = u[r];
        _Pragma("unroll")
        for (int r = 0; r < RR; ++r) v[r] = fft::cmul(v[r], __ldg(Ft + at + r * step));
        fft::dft_small<RR, 1>(v);
        _Pragma("unroll")
        for (int r = 0; r < RR; ++r) d[r * w] = v[r];
      });
      last_stage<W, RR, -1>(p, sm + tile, l, slot, [&](int q, float2(&v)[RR], float2* d) {
        const int64_t at = col + out_base(p, q) * row_s;
        _Pragma("unroll")
        for (int r = 0; r < RR; ++r) v[r] = fft::cmul(v[r], __ldg(Ft + at + r * step));
        fft::dft_small<RR, 1>(v);
        _Pragma("unroll")
        for (int r = 0; r < RR; ++r) d[r * w] = v[r];
      });
    }));
    __syncthreads();
    for (int s = p.ns - 2; s >= 1; --s) {
      TM_RADIX(p.r[s], ({
        mid_adjoint<W, RR>(p, s, sm, tw, l, slot);
        mid_adjoint<W, RR>(p, s, sm + tile, tw, l, slot);
        mid_adjoint<W, RR>(p, s, sm + 2 * tile, tw, l, slot);
      }));
      __syncthreads();
    }
    const int64_t h0 = b * hl.sb + k1 * hl.sr + k2;
    TM_RADIX(p.r[0], ({
      first_adjoint<W, RR>(p, sm, tw, l, slot,
                           [&](int q) { return output(Hm + h0 + q * hl.sx); });
      first_adjoint<W, RR>(p, sm + 2 * tile, tw, l, slot,
                           [&](int q) { return output(Hm2 + h0 + q * hl.sx); });
      first_adjoint<W, RR>(p, sm + tile, tw, l, slot,
                           [&](int q) { return output(Ht + h0 + q * hl.sx); });
    }));
  }
}

}  // namespace

int gen_prepare_xflc(const GenConfig& c, bool half) {
  TM_STORE(half, TM_LINES(c.x.plan, TM_TRY((raise(gen_xpass_flc_kernel<WW, HT>)))));
  return TM_OK;
}

int gen_xpass_flc(const GenConfig& c, const float2* Gt, const float2* Gm, const float2* Ft,
                  const float2* Ft2, int nb, int t0, int n1, int h2, int hp, const float4* tw0,
                  float scale, void* Ht, bool half, float2* Hm, float2* Hm2, const HLayout& hl,
                  cudaStream_t st) {
  const int per = rotations_per_cta((int64_t)(hp / c.x.plan.w) * n1, nb);
  const dim3 g(hp / c.x.plan.w, n1, (unsigned)ceil_div(nb, per));
  TM_STORE(half, TM_LINES(c.x.plan, (gen_xpass_flc_kernel<WW, HT><<<g, c.x.threads(), c.x.smem, st>>>(
                                    Gt, Gm, Ft, Ft2, nb, per, t0, n1, h2, c.x.plan, tw0,
                                    scale, static_cast<HT*>(Ht), Hm, Hm2, hl))));
  return check_launch("gen_xpass_flc_kernel");
}

}  // namespace tmb
