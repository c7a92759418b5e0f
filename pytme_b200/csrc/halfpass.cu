// Template rows, x pass and y pass of mixed-precision plans, whose spectra are stored as half2.
//
// A plan of mixed precision rounds its spectra to half after the x and after the y pass (and,
// for the tensor-core x pass, the template rows), and a rounding turns a difference in the
// last FP32 bit into one of 2^-11: transforms that round otherwise in FP32 move a score map by
// 1e-5 to 5e-5 of its norm and single voxels by 1e-3. So these plans keep their transforms,
// bit for bit; FP32 plans, and what a mixed plan keeps in FP32 (the FLC statistics), take the
// line FFTs of genpass.cuh.
//
// Power-of-two axes use the register-resident columns of colfft.cuh, other 5-smooth ones the
// shared-memory Stockham of fft_smem.cuh.
#include "halfpass.cuh"

#include <cuda_fp16.h>

#include <algorithm>
#include <cmath>
#include <type_traits>

#include "colfft.cuh"
#include "common.cuh"
#include "fft_smem.cuh"

namespace tmb {

using fft::LinePlan;

namespace {

LinePlan make_line_plan(int n) {
  LinePlan p{};
  p.n = n;
  int m = n, e2 = 0;
  while (m % 2 == 0) { m /= 2; ++e2; }
  int k = 0;
  int eights = e2 / 3, rem = e2 % 3;
  if (rem == 1 && eights > 0) { eights -= 1; p.radix[k++] = 4; p.radix[k++] = 4; }
  else if (rem == 1) { p.radix[k++] = 2; }
  else if (rem == 2) { p.radix[k++] = 4; }
  for (int i = 0; i < eights; ++i) p.radix[k++] = 8;
  for (int q : {3, 5, 7, 11, 13}) {
    while (m % q == 0) { m /= q; p.radix[k++] = q; }
  }
  p.npass = (m == 1) ? k : -1;
  return p;
}

// ------------------------------------------------------------------ storage types
template <typename T> struct Store;
template <> struct Store<float2> {
  static __device__ __forceinline__ float2 load(const float2* p) { return *p; }
  static __device__ __forceinline__ void store(float2* p, float2 v) { *p = v; }
};
template <> struct Store<__half2> {
  static __device__ __forceinline__ float2 load(const __half2* p) { return __half22float2(*p); }
  static __device__ __forceinline__ void store(__half2* p, float2 v) { *p = __float22half2_rn(v); }
};

// Asynchronous global -> shared copies (cp.async): the next tile is staged in shared
// memory while the current one is transformed. Each thread later reads back only the
// elements it copied, so a thread-local wait_group suffices.
template <int BYTES>
__device__ __forceinline__ void cp_async(void* smem, const void* gmem) {
  const unsigned s = (unsigned)__cvta_generic_to_shared(smem);
  if constexpr (BYTES == 4)
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;\n" ::"r"(s), "l"(gmem));
  else
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8;\n" ::"r"(s), "l"(gmem));
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::); }
template <int PENDING>
__device__ __forceinline__ void cp_async_wait() {
  asm volatile("cp.async.wait_group %0;\n" ::"n"(PENDING));
}

constexpr int kThreads = 512;
constexpr int kMaxE = 8;             // complex elements per thread in a line-FFT tile
constexpr int kTile = kThreads * kMaxE;  // elements per tile (4096)

// ------------------------------------------------------------------ K1: template z/y
// grid (ceil(h2/W), t0, B); tile: n1 lines-fast rows x W lines (k2).
__global__ void __launch_bounds__(kThreads, 1)
tmpl_zy_kernel(const float* __restrict__ tmpl, int t0, int t1, int t2, int n1, int n2, int h2,
               int W, LinePlan p1, const float2* __restrict__ tw1_g, const float2* __restrict__ tw2_g,
               float2* __restrict__ G) {
  extern __shared__ float4 smem_raw[];
  float2* tw1 = reinterpret_cast<float2*>(smem_raw);
  float2* tw2 = tw1 + n1;
  float2* buf = tw2 + n2;
  float* plane = reinterpret_cast<float*>(buf + (int64_t)n1 * W);
  const int tid = threadIdx.x;
  const int k2_0 = blockIdx.x * W;
  const int x = blockIdx.y;
  const int b = blockIdx.z;
  for (int i = tid; i < n1; i += kThreads) tw1[i] = tw1_g[i];
  for (int i = tid; i < n2; i += kThreads) tw2[i] = tw2_g[i];
  const float* src = tmpl + ((int64_t)b * t0 + x) * t1 * t2;
  for (int i = tid; i < t1 * t2; i += kThreads) plane[i] = src[i];
  __syncthreads();
  // G1[y][k2] = sum_z plane[y][z] * exp(-2 pi i z k2 / n2), rows y >= t1 are zero
  for (int e = tid; e < n1 * W; e += kThreads) {
    int y = e / W, l = e % W;
    int k2 = k2_0 + l;
    float2 acc = make_float2(0.f, 0.f);
    if (y < t1 && k2 < h2) {
      const float* row = plane + y * t2;
      int idx = 0;
      for (int z = 0; z < t2; ++z) {
        float v = row[z];
        float2 w = tw2[idx];
        acc.x += v * w.x;
        acc.y += v * w.y;
        idx += k2;
        if (idx >= n2) idx -= n2;
      }
    }
    buf[e] = acc;
  }
  __syncthreads();
  fft::fft_lines<-1, kMaxE, true>(buf, p1, W, 1, W, tw1, n1, tid, kThreads);
  float2* dst = G + ((int64_t)b * t0 + x) * n1 * h2;
  for (int e = tid; e < n1 * W; e += kThreads) {
    int k1 = e / W, l = e % W;
    int k2 = k2_0 + l;
    if (k2 < h2) dst[(int64_t)k1 * h2 + k2] = buf[e];
  }
}

// ------------------------------------------------------------------ K2: x pass
// grid (ceil(h2/W), n1); loops over the B rotations of the group.
template <typename HT>
__global__ void __launch_bounds__(kThreads, 1)
xpass_kernel(const float2* __restrict__ G, const float2* __restrict__ Ft, int B, int t0, int n0,
             int n1, int h2, int W, LinePlan p0, const float2* __restrict__ tw0_g, float scale,
             HT* __restrict__ H, int hp) {
  extern __shared__ float4 smem_raw[];
  float2* tw0 = reinterpret_cast<float2*>(smem_raw);
  float2* buf = tw0 + n0;
  const int tid = threadIdx.x;
  const int k2_0 = blockIdx.x * W;
  const int k1 = blockIdx.y;
  for (int i = tid; i < n0; i += kThreads) tw0[i] = tw0_g[i];
  const int tile = n0 * W;
  // target-spectrum tile: re-read through L1 for every rotation of the group
  const float2* ft_col = Ft + (int64_t)k1 * h2 + k2_0;
  const int64_t ft_row = (int64_t)n1 * h2;
  const int64_t SH = (int64_t)n0 * n1 * hp;
  for (int b = 0; b < B; ++b) {
    const float2* g = G + (int64_t)b * t0 * n1 * h2;
    for (int e = tid; e < tile; e += kThreads) {
      int x = e / W, l = e % W;
      int k2 = k2_0 + l;
      float2 v = make_float2(0.f, 0.f);
      if (x < t0 && k2 < h2) v = g[((int64_t)x * n1 + k1) * h2 + k2];
      buf[e] = v;
    }
    __syncthreads();
    fft::fft_lines<-1, kMaxE, true>(buf, p0, W, 1, W, tw0, n0, tid, kThreads);
    for (int e = tid; e < tile; e += kThreads) {
      int k0 = e / W, l = e % W;
      float2 f = make_float2(0.f, 0.f);
      if (k2_0 + l < h2) f = __ldg(ft_col + k0 * ft_row + l);
      buf[e] = fft::cmul(buf[e], make_float2(f.x * scale, f.y * scale));
    }
    __syncthreads();
    fft::fft_lines<1, kMaxE, true>(buf, p0, W, 1, W, tw0, n0, tid, kThreads);
    HT* h = H + (int64_t)b * SH;
    for (int e = tid; e < tile; e += kThreads) {
      int x = e / W, l = e % W;
      int k2 = k2_0 + l;
      if (k2 < h2) Store<HT>::store(h + ((int64_t)x * n1 + k1) * hp + k2, buf[e]);
    }
    __syncthreads();
  }
}

// ------------------------------------------------------------------ K3: y pass
// grid (ceil(h2/W), n0, B): inverse FFT along axis 1, in place.
template <typename HT>
__global__ void __launch_bounds__(kThreads, 1)
ypass_kernel(HT* __restrict__ H, int n0, int n1, int h2, int W, LinePlan p1,
             const float2* __restrict__ tw1_g, int hp) {
  extern __shared__ float4 smem_raw[];
  float2* tw1 = reinterpret_cast<float2*>(smem_raw);
  float2* buf = tw1 + n1;
  const int tid = threadIdx.x;
  const int k2_0 = blockIdx.x * W;
  const int x = blockIdx.y;
  const int b = blockIdx.z;
  for (int i = tid; i < n1; i += kThreads) tw1[i] = tw1_g[i];
  const int tile = n1 * W;
  HT* h = H + (int64_t)b * n0 * n1 * hp + (int64_t)x * n1 * hp;
  for (int e = tid; e < tile; e += kThreads) {
    int y = e / W, l = e % W;
    int k2 = k2_0 + l;
    buf[e] = (k2 < h2) ? Store<HT>::load(h + (int64_t)y * hp + k2) : make_float2(0.f, 0.f);
  }
  __syncthreads();
  fft::fft_lines<1, kMaxE, true>(buf, p1, W, 1, W, tw1, n1, tid, kThreads);
  for (int e = tid; e < tile; e += kThreads) {
    int y = e / W, l = e % W;
    int k2 = k2_0 + l;
    if (k2 < h2) Store<HT>::store(h + (int64_t)y * hp + k2, buf[e]);
  }
}

// ------------------------------------------------------------------ register-resident passes
// Power-of-two axis lengths use the column codelet of colfft.cuh: T = N/8 threads
// per column, W columns per CTA (thread id = t*W + l, so a warp spans W columns and
// each global row segment of W elements is one contiguous access).

// Stage 0 of the forward DIF when only rows [0, nz) of the column are non-zero and
// nz <= T: the radix-8 DFT of a single non-zero input is that input, so output j is
// x[t] * W_N^(j*t).
template <int N>
__device__ __forceinline__ void stage0_single(float2 (&v)[8], int t, const float2* tw) {
  const float2 w1 = tw[t];
  float2 x = v[0];
  v[0] = x;
#pragma unroll
  for (int j = 1; j < 8; ++j) {
    x = fft::cmul(x, w1);
    v[j] = x;
  }
}

// The same for the FLC numerators, whose powers are contracted the other way round: the
// imaginary part of x * w as fma(x.x, w.y, x.y * w.x). (stage0_single leaves the choice to
// the compiler, which takes fma(x.y, w.x, x.x * w.y) in the x pass of CC and
// FLCSphericalMask and took this one in the kernel that FLC had of its own.)
template <int N>
__device__ __forceinline__ void stage0_single_flc(float2 (&v)[8], int t, const float2* tw) {
  const float2 w1 = tw[t];
  float2 x = v[0];
#pragma unroll
  for (int j = 1; j < 8; ++j) {
    x = make_float2(__fmaf_rn(x.x, w1.x, -__fmul_rn(x.y, w1.y)),
                    __fmaf_rn(x.x, w1.y, __fmul_rn(x.y, w1.x)));
    v[j] = x;
  }
}

template <int N, int W, int DIR>
__device__ __forceinline__ void dif_rest(float2 (&v)[8], float2* sm, const float2* tw, int l,
                                         int t) {
  constexpr int NS = colfft::num_stages(N);
  colfft::store_stage<N, W, 0>(v, sm, l, t);
  __syncthreads();
  if constexpr (NS > 1) {
    colfft::load_stage<N, W, 1>(v, sm, l, t);
    colfft::dif_stage_regs<N, 1, DIR>(v, t, tw);
  }
  if constexpr (NS > 2) {
    colfft::store_stage<N, W, 1>(v, sm, l, t);
    __syncthreads();
    colfft::load_stage<N, W, 2>(v, sm, l, t);
    colfft::dif_stage_regs<N, 2, DIR>(v, t, tw);
  }
  if constexpr (NS > 3) {
    colfft::store_stage<N, W, 2>(v, sm, l, t);
    __syncthreads();
    colfft::load_stage<N, W, 3>(v, sm, l, t);
    colfft::dif_stage_regs<N, 3, DIR>(v, t, tw);
  }
}

// K1': template rows -> G. grid (ceil(h2/W), t0, B); N = n1.
template <int N, int W, typename GT = float2>
__global__ void __launch_bounds__(N / 8 * W, 1)
tmpl_zy_reg_kernel(const float* __restrict__ tmpl, int t0, int t1, int t2, int n2, int h2,
                   const float2* __restrict__ tw1_g, const float2* __restrict__ tw2_g,
                   GT* __restrict__ G) {
  constexpr int T = N / 8;
  constexpr int NT = T * W;
  extern __shared__ float4 smem_raw[];
  float2* tw1 = reinterpret_cast<float2*>(smem_raw);
  float2* sm = tw1 + N;
  float2* tw2 = sm + colfft::smem_elems<N>(W);
  float* plane = reinterpret_cast<float*>(tw2 + n2);
  const int tid = threadIdx.x, l = tid % W, t = tid / W;
  const int k2 = blockIdx.x * W + l;
  const int x = blockIdx.y, b = blockIdx.z;
  for (int i = tid; i < N; i += NT) tw1[i] = tw1_g[i];
  for (int i = tid; i < n2; i += NT) tw2[i] = tw2_g[i];
  const float* src = tmpl + ((int64_t)b * t0 + x) * t1 * t2;
  for (int i = tid; i < t1 * t2; i += NT) plane[i] = src[i];
  __syncthreads();
  float2 v[8];
#pragma unroll
  for (int r = 0; r < 8; ++r) {
    const int y = t + T * r;
    float2 acc = make_float2(0.f, 0.f);
    if (y < t1 && k2 < h2) {
      const float* row = plane + y * t2;
      int idx = 0;
      for (int z = 0; z < t2; ++z) {
        const float a = row[z];
        const float2 w = tw2[idx];
        acc.x += a * w.x;
        acc.y += a * w.y;
        idx += k2;
        if (idx >= n2) idx -= n2;
      }
    }
    v[r] = acc;
  }
  if (t1 <= T) stage0_single<N>(v, t, tw1);
  else colfft::dif_stage_regs<N, 0, -1>(v, t, tw1);
  dif_rest<N, W, -1>(v, sm, tw1, l, t);
  if (k2 < h2) {
    GT* dst = G + ((int64_t)b * t0 + x) * N * h2;
    constexpr int R = colfft::stage_radix(N, colfft::num_stages(N) - 1);
#pragma unroll
    for (int i = 0; i < 8 / R; ++i)
#pragma unroll
      for (int r = 0; r < R; ++r) {
        const int k1 = colfft::out_index<N>(t, i, r);
        Store<GT>::store(dst + (int64_t)k1 * h2 + k2, v[i * R + r]);
      }
  }
}

// K2': x pass. grid (ceil(h2/W), n1); N = n0; loops over the rotations of the group.
template <int N, int W, typename HT, bool FLC = false>
__global__ void __launch_bounds__(N / 8 * W, 1024 / (N / 8 * W))
xpass_reg_kernel(const float2* __restrict__ G, const float2* __restrict__ Ft, int B, int t0,
                 int n1, int h2, const float2* __restrict__ tw0_g, float scale,
                 HT* __restrict__ H, int hp) {
  constexpr int T = N / 8;
  constexpr int NT = T * W;
  constexpr int R = colfft::stage_radix(N, colfft::num_stages(N) - 1);
  extern __shared__ float4 smem_raw[];
  float2* tw = reinterpret_cast<float2*>(smem_raw);
  float2* sm = tw + N;
  const int tid = threadIdx.x, l = tid % W, t = tid / W;
  const int k2 = blockIdx.x * W + l;
  const int k1 = blockIdx.y;
  const bool valid = k2 < h2;
  for (int i = tid; i < N; i += NT) tw[i] = tw0_g[i];
  // offsets of the target-spectrum values this thread multiplies (through L1, reused
  // by every rotation of the group)
  const int64_t col = (int64_t)k1 * h2 + k2;
  const int64_t row = (int64_t)n1 * h2;
  const float2* fb = Ft + (int64_t)colfft::out_index<N>(t, 0, 0) * row + col;
  __syncthreads();
  const int64_t SH = (int64_t)N * n1 * hp, rowH = (int64_t)n1 * hp;
  const int64_t colH = (int64_t)k1 * hp + k2;
  for (int b = 0; b < B; ++b) {
    const float2* g = G + (int64_t)b * t0 * row + col;
    float2 v[8];
#pragma unroll
    for (int r = 0; r < 8; ++r) {
      const int x = t + T * r;
      v[r] = (valid && x < t0) ? g[(int64_t)x * row] : make_float2(0.f, 0.f);
    }
    if (FLC && t0 <= T) stage0_single_flc<N>(v, t, tw);
    else if (t0 <= T) stage0_single<N>(v, t, tw);
    else colfft::dif_stage_regs<N, 0, -1>(v, t, tw);
    dif_rest<N, W, -1>(v, sm, tw, l, t);
#pragma unroll
    for (int i = 0; i < 8 / R; ++i)
#pragma unroll
      for (int r = 0; r < R; ++r) {
        // out_index(t, i, r) = out_index(t, i, 0) + r * N/R; out_index(t, i, 0) - out_index(t, 0, 0)
        // depends on i only through compile-time digits
        const int dk = colfft::out_index<N>(t, i, r) - colfft::out_index<N>(t, 0, 0);
        const float2 f = valid ? __ldg(fb + (int64_t)dk * row) : make_float2(0.f, 0.f);
        v[i * R + r] = fft::cmul(v[i * R + r], make_float2(f.x * scale, f.y * scale));
      }
    colfft::dif_adjoint<N, W>(v, sm, tw, l, t);
    if (valid) {
      HT* h = H + (int64_t)b * SH + colH;
#pragma unroll
      for (int r = 0; r < 8; ++r) Store<HT>::store(h + (int64_t)(t + T * r) * rowH, v[r]);
    }
  }
}

// K3': y pass (inverse FFT along axis 1, in place). grid (ceil(h2/W), ceil(n0/XP), B);
// each CTA walks XP consecutive x planes; the next plane's columns are staged in shared
// memory with cp.async while the current plane is transformed (each thread stages and
// later reads only its own elements, so a stage is reused without a barrier). The pass
// is bound by instruction issue and shared-memory traffic, not by loads in flight:
// three or four staged planes measured slower than two. N = n1.
constexpr int kYPlanes = 8;
constexpr int kYStages = 2;

template <int N, int W, typename HT>
__global__ void __launch_bounds__(N / 8 * W, 1024 / (N / 8 * W))
ypass_reg_kernel(HT* __restrict__ H, int n0, int h2, const float2* __restrict__ tw1_g, int hp,
                 int seg) {
  constexpr int T = N / 8;
  constexpr int NT = T * W;
  constexpr int R = colfft::stage_radix(N, colfft::num_stages(N) - 1);
  extern __shared__ float4 smem_raw[];
  float2* tw = reinterpret_cast<float2*>(smem_raw);
  float2* sm = tw + N;
  HT* stage = reinterpret_cast<HT*>(sm + colfft::smem_elems<N>(W));  // kYStages x N*W staging
  const int tid = threadIdx.x, l = tid % W, t = tid / W;
  const int k2 = blockIdx.x * W + l;
  const int x0 = blockIdx.y * kYPlanes, b = blockIdx.z;
  const int nx = min(kYPlanes, n0 - x0);
  const bool valid = k2 < h2;
  for (int i = tid; i < N; i += NT) tw[i] = tw1_g[i];
  HT* base = H + ((int64_t)b * n0 + x0) * N * hp + k2;
  const int64_t plane = (int64_t)N * hp;
  auto fetch = [&](int xi) {
    if (valid && xi < nx) {
      HT* dst = stage + (xi % kYStages) * N * W;
      const HT* src = base + (int64_t)xi * plane;
#pragma unroll
      for (int r = 0; r < 8; ++r)
        cp_async<sizeof(HT)>(dst + (t + T * r) * W + l, src + (int64_t)(t + T * r) * hp);
    }
    cp_async_commit();  // one group per plane, empty past the last
  };
#pragma unroll
  for (int xi = 0; xi < kYStages - 1; ++xi) fetch(xi);
  __syncthreads();  // twiddles
  for (int xi = 0; xi < nx; ++xi) {
    HT* cur = stage + (xi % kYStages) * N * W;
    fetch(xi + kYStages - 1);
    cp_async_wait<kYStages - 1>();  // plane xi landed
    float2 v[8];
#pragma unroll
    for (int r = 0; r < 8; ++r)
      v[r] = valid ? Store<HT>::load(cur + (t + T * r) * W + l) : make_float2(0.f, 0.f);
    colfft::dif_stage_regs<N, 0, 1>(v, t, tw);
    dif_rest<N, W, 1>(v, sm, tw, l, t);
    if constexpr (std::is_same<HT, __half2>::value) {
      if (seg) {
        // 32-byte segments [Re x 8 | Im x 8] of 8 consecutive k2 (the even/odd tensor-core
        // z pass's input): the 8 lanes holding one row's segment exchange values so each
        // stores one word, (Re, Re) of columns 2q, 2q+1 for q < 4, (Im, Im) after that
        const int q = l & 7, lane = threadIdx.x & 31;
        const int srcA = (lane & ~7) | ((2 * q) & 7);
        const uint32_t sel = q < 4 ? 0x5410u : 0x7632u;
        HT* h = base + (int64_t)xi * plane;
#pragma unroll
        for (int i = 0; i < 8 / R; ++i)
#pragma unroll
          for (int r = 0; r < R; ++r) {
            const int y = colfft::out_index<N>(t, i, r);
            const __half2 hv = __float22half2_rn(v[i * R + r]);
            uint32_t w = *reinterpret_cast<const uint32_t*>(&hv);
            const uint32_t a = __shfl_sync(0xffffffffu, w, srcA);
            const uint32_t b = __shfl_sync(0xffffffffu, w, srcA + 1);
            w = __byte_perm(a, b, sel);
            if (k2 < hp) *reinterpret_cast<uint32_t*>(h + (int64_t)y * hp) = w;
          }
        __syncthreads();  // the next plane's stage-0 stores reuse the exchange buffer
        continue;
      }
    }
    if (valid) {
      HT* h = base + (int64_t)xi * plane;
#pragma unroll
      for (int i = 0; i < 8 / R; ++i)
#pragma unroll
        for (int r = 0; r < R; ++r) {
          const int y = colfft::out_index<N>(t, i, r);
          Store<HT>::store(h + (int64_t)y * hp, v[i * R + r]);
        }
    }
    __syncthreads();  // the next plane's stage-0 stores reuse the exchange buffer
  }
}

template <int N>
constexpr int reg_lines() { return N >= 512 ? 8 : 16; }

template <int N>
size_t reg_smem_bytes(int n2, int t1, int t2, bool with_plane) {
  size_t b = sizeof(float2) * (N + colfft::smem_elems<N>(reg_lines<N>()));
  if (with_plane) b += sizeof(float2) * n2 + sizeof(float) * t1 * t2;
  return b;
}

template <int N, typename HT>
size_t ypass_smem_bytes() {
  return reg_smem_bytes<N>(0, 0, 0, false) + kYStages * sizeof(HT) * N * reg_lines<N>();
}

static bool reg_supported(int n) {
  return n == 64 || n == 128 || n == 256 || n == 512 || n == 1024;
}

#define TM_DISPATCH_N(n, CALL)                         \
  switch (n) {                      \
    case 64: { constexpr int NN = 64; CALL; } break;    \
    case 128: { constexpr int NN = 128; CALL; } break;  \
    case 256: { constexpr int NN = 256; CALL; } break;  \
    case 512: { constexpr int NN = 512; CALL; } break;  \
    case 1024: { constexpr int NN = 1024; CALL; } break; \
    default: break;                 \
  }

int optin_max() {
  int dev = 0, v = 48 * 1024;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&v, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
  return v;
}

template <class K>
int raise(K kernel) {
  return cuda_status(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                          optin_max()),
                     "shared memory limit");
}

}  // namespace

HalfConfig half_config(int n0, int n1, int n2, int h2, int t1, int t2) {
  HalfConfig c;
  c.reg0 = reg_supported(n0);
  c.reg1 = reg_supported(n1);
  c.p0 = make_line_plan(n0);
  c.p1 = make_line_plan(n1);
  c.w0 = std::max(1, std::min(h2, kTile / n0));
  c.w1 = std::max(1, std::min(h2, kTile / n1));
  c.smt = sizeof(float2) * (n1 + n2 + (size_t)n1 * c.w1) + sizeof(float) * t1 * t2;
  c.smx = sizeof(float2) * (n0 + (size_t)n0 * c.w0);
  c.smy = sizeof(float2) * (n1 + (size_t)n1 * c.w1);
  if (c.reg1) {
    size_t zy = 0;
    TM_DISPATCH_N(n1, (zy = reg_smem_bytes<NN>(n2, t1, t2, true)));
    if (zy > 200 * 1024) c.reg1 = false;
  }
  return c;
}

int half_prepare(const HalfConfig& c, int n0, int n1) {
  if (c.reg0) {
    TM_DISPATCH_N(n0, TM_TRY((raise(xpass_reg_kernel<NN, reg_lines<NN>(), __half2>))));
    TM_DISPATCH_N(n0, TM_TRY((raise(xpass_reg_kernel<NN, reg_lines<NN>(), __half2, true>))));
  } else {
    TM_TRY(raise(xpass_kernel<__half2>));
  }
  if (c.reg1) {
    TM_DISPATCH_N(n1, TM_TRY((raise(ypass_reg_kernel<NN, reg_lines<NN>(), __half2>))));
    TM_DISPATCH_N(n1, TM_TRY((raise(tmpl_zy_reg_kernel<NN, reg_lines<NN>(), float2>))));
    TM_DISPATCH_N(n1, TM_TRY((raise(tmpl_zy_reg_kernel<NN, reg_lines<NN>(), __half2>))));
  } else {
    TM_TRY(raise(ypass_kernel<__half2>));
    TM_TRY(raise(tmpl_zy_kernel));
  }
  return TM_OK;
}

int half_template(const HalfConfig& c, const float* tmpl, int nb, int t0, int t1, int t2, int n1,
                  int n2, int h2, const float2* tw1, const float2* tw2, void* G, bool half_g,
                  cudaStream_t st) {
  if (c.reg1) {
    TM_DISPATCH_N(n1, ({
      constexpr int W = reg_lines<NN>();
      const dim3 g((unsigned)ceil_div(h2, W), t0, nb);
      const size_t smem = reg_smem_bytes<NN>(n2, t1, t2, true);
      if (half_g)
        tmpl_zy_reg_kernel<NN, W, __half2><<<g, NN / 8 * W, smem, st>>>(
            tmpl, t0, t1, t2, n2, h2, tw1, tw2, static_cast<__half2*>(G));
      else
        tmpl_zy_reg_kernel<NN, W, float2><<<g, NN / 8 * W, smem, st>>>(
            tmpl, t0, t1, t2, n2, h2, tw1, tw2, static_cast<float2*>(G));
    }));
  } else {
    const dim3 g((unsigned)ceil_div(h2, c.w1), t0, nb);
    tmpl_zy_kernel<<<g, kThreads, c.smt, st>>>(tmpl, t0, t1, t2, n1, n2, h2, c.w1, c.p1, tw1, tw2,
                                               static_cast<float2*>(G));
  }
  return check_launch("template pass");
}

int half_xpass(const HalfConfig& c, const float2* G, const float2* Ft, int nb, int t0, int n0,
               int n1, int h2, int hp, const float2* tw0, float scale, void* H, bool flc,
               cudaStream_t st) {
  if (c.reg0) {
    TM_DISPATCH_N(n0, ({
      constexpr int W = reg_lines<NN>();
      const dim3 g((unsigned)ceil_div(h2, W), n1);
      const size_t smem = reg_smem_bytes<NN>(0, 0, 0, false);
      if (flc)
        xpass_reg_kernel<NN, W, __half2, true><<<g, NN / 8 * W, smem, st>>>(
            G, Ft, nb, t0, n1, h2, tw0, scale, static_cast<__half2*>(H), hp);
      else
              xpass_reg_kernel<NN, W, __half2><<<g, NN / 8 * W, smem, st>>>(
            G, Ft, nb, t0, n1, h2, tw0, scale, static_cast<__half2*>(H), hp);
    }));
  } else {
    const dim3 g((unsigned)ceil_div(h2, c.w0), n1);
    xpass_kernel<__half2><<<g, kThreads, c.smx, st>>>(G, Ft, nb, t0, n0, n1, h2, c.w0, c.p0, tw0,
                                                     scale, static_cast<__half2*>(H), hp);
  }
  return check_launch("x pass");
}

int half_ypass(const HalfConfig& c, void* H, int nb, int n0, int n1, int h2, int hp,
               const float2* tw1, bool seg, cudaStream_t st) {
  __half2* h = static_cast<__half2*>(H);
  if (c.reg1) {
    TM_DISPATCH_N(n1, ({
      constexpr int W = reg_lines<NN>();
      const dim3 g((unsigned)ceil_div(h2, W), (unsigned)ceil_div(n0, kYPlanes), nb);
      ypass_reg_kernel<NN, W, __half2><<<g, NN / 8 * W, ypass_smem_bytes<NN, __half2>(), st>>>(
          h, n0, h2, tw1, hp, seg ? 1 : 0);
    }));
  } else {
    const dim3 g((unsigned)ceil_div(h2, c.w1), n0, nb);
    ypass_kernel<__half2><<<g, kThreads, c.smy, st>>>(h, n0, n1, h2, c.w1, c.p1, tw1, hp);
  }
  return check_launch("y pass");
}

}  // namespace tmb
