// fftconv.cu -- the z pass of the periodic Poisson solve of POFFT3D
// (poisson.f:98-249) for NX in {64, 128, 256, 512}.
//
// The solve runs as three passes over the half spectrum: the library's
// batched 2-D R2C of every (copy, z) plane, then k_fft_z_green (FFT along z,
// the Green's multiply KKK/NX^3 of MOMENTO's table, inverse FFT along z, in
// place, one pass), then the library's 2-D C2R.  Against a library 3-D
// R2C, a separate multiply and a 3-D C2R, the z transforms and the multiply
// share one read and one write of the spectrum.
//
// A line of N = V T values is transformed by T threads in two register
// passes with one exchange through shared memory.  Thread s holds elements
// s + T n1 (n1 < V): a V-point FFT over n1 gives A[k1], the exchange hands
// thread k1 mod T the values A_s[k1] of every s, which it turns by W_N^(s k1)
// and transforms over s into the frequencies k1 + V k2.  The Green's factor is
// applied there, and the same steps undone in reverse order return natural
// order; each thread writes its groups back where it read them, so the
// exchange buffer needs two barriers in all.  Register FFTs are decimation in
// frequency forward (output in bit-reversed order) and decimation in time
// back (input in bit-reversed order), so nothing is permuted.  Twiddles W_N^j
// are a table computed on the host in double precision.  The result equals an
// FFT-based solve within float32 rounding (not bit for bit a library's).
#include <cuda_runtime.h>
#include <math.h>

#include <vector>

#include "common.cuh"

namespace {

__device__ __forceinline__ float2 cadd(float2 a, float2 b) { return make_float2(a.x + b.x, a.y + b.y); }
__device__ __forceinline__ float2 csub(float2 a, float2 b) { return make_float2(a.x - b.x, a.y - b.y); }
// complex product with fused multiply-adds (two roundings per part)
__device__ __forceinline__ float2 cmul(float2 a, float2 b) {
  return make_float2(__fmaf_rn(a.x, b.x, -__fmul_rn(a.y, b.y)), __fmaf_rn(a.x, b.y, __fmul_rn(a.y, b.x)));
}
__device__ __forceinline__ float2 conjf2(float2 a) { return make_float2(a.x, -a.y); }

__host__ __device__ constexpr int ilog2(int v) { return v <= 1 ? 0 : 1 + ilog2(v >> 1); }
__host__ __device__ constexpr int brev_c(int p, int bits) {
  int r = 0;
  for (int b = 0; b < bits; b++)
    if ((p >> b) & 1) r |= 1 << (bits - 1 - b);
  return r;
}

// cos and sin of 2 pi j / n (0 <= j <= n/2) at compile time: the Taylor
// series of the angle folded into [0, pi/4]
__host__ __device__ constexpr double taylor(double x, bool sine) {
  double term = sine ? x : 1.0, sum = term;
  for (int k = sine ? 2 : 1; k < 40; k += 2) {
    term *= -x * x / (double)(k * (k + 1));
    sum += term;
  }
  return sum;
}
__host__ __device__ constexpr double cos_turn(int j, int n);
__host__ __device__ constexpr double sin_turn(int j, int n) {
  return 4 * j > n ? sin_turn(n / 2 - j, n)
                   : (8 * j > n ? taylor(6.283185307179586476925 * (n / 4 - j) / n, false)
                                : taylor(6.283185307179586476925 * j / n, true));
}
__host__ __device__ constexpr double cos_turn(int j, int n) {
  return 4 * j > n ? -cos_turn(n / 2 - j, n)
                   : (8 * j > n ? taylor(6.283185307179586476925 * (n / 4 - j) / n, true)
                                : taylor(6.283185307179586476925 * j / n, false));
}

// v W_M^j (INV: v W_M^-j) for constant j < M/2
template <int M, int J, bool INV>
__device__ __forceinline__ float2 turn(float2 v) {
  if constexpr (J == 0) {
    return v;
  } else if constexpr (4 * J == M) {
    return INV ? make_float2(-v.y, v.x) : make_float2(v.y, -v.x);
  } else {
    constexpr float c = (float)cos_turn(J, M), s = (float)sin_turn(J, M);
    return cmul(v, make_float2(c, INV ? s : -s));
  }
}

// One stage of the register FFT: blocks of 2H, butterflies J, J + H.
template <int R, int H, bool INV, int J>
__device__ __forceinline__ void stage(float2 (&v)[R]) {
  if constexpr (J < H) {
#pragma unroll
    for (int b = 0; b < R; b += 2 * H) {
      const float2 a = v[b + J];
      if (!INV) {
        const float2 c = v[b + J + H];
        v[b + J] = cadd(a, c);
        v[b + J + H] = turn<2 * H, J, false>(csub(a, c));
      } else {
        const float2 c = turn<2 * H, J, true>(v[b + J + H]);
        v[b + J] = cadd(a, c);
        v[b + J + H] = csub(a, c);
      }
    }
    stage<R, H, INV, J + 1>(v);
  }
}

// R-point DFT in registers, sign -1: natural order in, v[p] = X[brev(p)] out.
template <int R, int H = R / 2>
__device__ __forceinline__ void fft_reg(float2 (&v)[R]) {
  if constexpr (H >= 1) {
    stage<R, H, false, 0>(v);
    fft_reg<R, H / 2>(v);
  }
}
// The unnormalised inverse: v[p] = X[brev(p)] in, natural order out.
template <int R, int H = 1>
__device__ __forceinline__ void ifft_reg(float2 (&v)[R]) {
  if constexpr (H < R) {
    stage<R, H, true, 0>(v);
    ifft_reg<R, 2 * H>(v);
  }
}

// N = V T: V values a thread, T threads a line, 16 lines (128-byte runs of a
// plane's rows) a CTA.  V and T near sqrt(N) keep the exchanges at one.
template <int N>
struct Geo {
  static constexpr int NCOL = N / 2 + 1;  // kx = 0..N/2
  static constexpr int TY = 16;           // lines per tile
  static constexpr int T = N >= 256 ? 16 : 8;
  static constexpr int V = N / T;
  static constexpr int ZT = TY * T;  // threads
  static constexpr int MINB = N == 512 ? 3 : (N == 256 ? 4 : 8);  // CTAs an SM: 80 and 64 registers
  static constexpr size_t ZSMEM = sizeof(float2) * (size_t)TY * N;
};

}  // namespace

// The z pass: a tile is TY consecutive values of one copy's (ky, kx) plane
// ([copy][z][ky][kx], NX/2+1 values per row, as the library's 2-D R2C leaves
// it), all NX z, in place: FFT along z, the Green's factor, inverse FFT
// along z.  KKK / N^3 = (-DEL2 / N^3) x 1 / (s2[kx] + s2[ky] + s2[kz])
// (denominator 1e30 at the origin; the reciprocal correctly rounded), on
// both parts.  One read and one write of the spectrum: 1.08 GB in 0.25 ms at
// 8 x 256^3 (0.65 of the measured copy rate) and in 0.32 ms at 512^3; with one
// warp a line and the FFT across lanes by shuffles, 0.44 and 0.54 ms, held by
// the shuffle queue.  What is left is the instruction issue of the two register
// transforms.
template <int N>
__global__ void __launch_bounds__(Geo<N>::ZT, Geo<N>::MINB)
k_fft_z_green(float2* __restrict__ spec, const float2* __restrict__ tw, const float* __restrict__ s2,
              float del2, float inv_n3) {
  using G = Geo<N>;
  constexpr int T = G::T, V = G::V, TY = G::TY, QT = N * G::NCOL / TY;
  extern __shared__ float2 sm[];  // [k1][s][line]
  const int j = threadIdx.x % TY, s = threadIdx.x / TY;
  const int64_t t = blockIdx.x;
  const int qq = (int)(t % QT) * TY + j;
  const int64_t zstride = (int64_t)G::NCOL * N;
  float2* base = spec + (t / QT) * N * zstride + qq;
  float2* own = sm + s * TY + j;
  {
    float2 v[V];
#pragma unroll
    for (int n1 = 0; n1 < V; n1++) v[n1] = base[(int64_t)(s + T * n1) * zstride];
    fft_reg<V>(v);
#pragma unroll
    for (int p = 0; p < V; p++) own[brev_c(p, ilog2(V)) * T * TY] = v[p];
  }
  __syncthreads();
  const int kx = qq % G::NCOL, ky = qq / G::NCOL;
  const float scale = __fmul_rn(-del2, inv_n3);
  const float sxy = __fadd_rn(__ldg(s2 + kx), __ldg(s2 + ky));
#pragma unroll
  for (int g = 0; g < V / T; g++) {
    const int k1 = s + T * g;
    float2* row = sm + k1 * T * TY + j;
    float2 u[T];
#pragma unroll
    for (int q = 0; q < T; q++) u[q] = cmul(row[q * TY], __ldg(tw + q * k1));
    fft_reg<T>(u);
#pragma unroll
    for (int p = 0; p < T; p++) {
      const int kz = k1 + V * brev_c(p, ilog2(T));
      const float den = (kx == 0 && ky == 0 && kz == 0) ? 1.0e30f : __fadd_rn(sxy, __ldg(s2 + kz));
      const float f = __fmul_rn(scale, __frcp_rn(den));
      u[p] = make_float2(__fmul_rn(u[p].x, f), __fmul_rn(u[p].y, f));
    }
    ifft_reg<T>(u);
#pragma unroll
    for (int q = 0; q < T; q++) row[q * TY] = cmul(u[q], conjf2(__ldg(tw + q * k1)));
  }
  __syncthreads();
  float2 v[V];
#pragma unroll
  for (int p = 0; p < V; p++) v[p] = own[brev_c(p, ilog2(V)) * T * TY];
  ifft_reg<V>(v);
#pragma unroll
  for (int n1 = 0; n1 < V; n1++) base[(int64_t)(s + T * n1) * zstride] = v[n1];
}

// W_N^j = exp(-2 pi i j / N), j < N, in double then rounded; exact at the
// quarter turns.  Kept on the context per N.
static int twiddles(asohf_ctx* c, int n, const float2** out) {
  if (c->tw_n != n) {
    ASOHF_CUDA(cudaStreamSynchronize(c->stream));
    cudaFree(c->d_tw);
    c->d_tw = nullptr;
    c->tw_n = 0;
    std::vector<float2> h((size_t)n);
    const double two_pi = 2.0 * acos(-1.0);
    for (int j = 0; j < n; j++) {
      const double a = two_pi * (double)j / (double)n;
      h[j] = make_float2((float)cos(a), (float)-sin(a));
    }
    h[0] = make_float2(1.f, 0.f);
    h[n / 4] = make_float2(0.f, -1.f);
    h[n / 2] = make_float2(-1.f, 0.f);
    h[3 * n / 4] = make_float2(0.f, 1.f);
    cudaError_t e = cudaMalloc(&c->d_tw, sizeof(float2) * (size_t)n);
    ASOHF_CUDA(e);
    ASOHF_CHECK(upload_table(c, c->d_tw, h.data(), sizeof(float2) * (size_t)n));
    c->tw_n = n;
  }
  *out = c->d_tw;
  return ASOHF_OK;
}

// The z pass on the context stream, on a half spectrum in the library 2-D
// transform's layout ([copy][z][ky][kx], NX/2+1 values per row, batch * NX
// planes): ASOHF_ERR_UNSUPPORTED unless NX is one of the sizes above and
// spec is 8-byte aligned.
int fftconv_z_green_2d(asohf_ctx* c, int nx, int batch, void* spec, const float* s2, float del2, float inv_n3) {
  if (nx != 64 && nx != 128 && nx != 256 && nx != 512) return ASOHF_ERR_UNSUPPORTED;
  if ((uintptr_t)spec & 7u) return ASOHF_ERR_UNSUPPORTED;
  const float2* tw;
  ASOHF_CHECK(twiddles(c, nx, &tw));
  float2* sp = (float2*)spec;
  int kt_ = ktime_begin(c, "fft_z_green");
  switch (nx) {
#define ZCASE(NN)                                                                                       \
  case NN:                                                                                              \
    ASOHF_CUDA(cudaFuncSetAttribute(k_fft_z_green<NN>, cudaFuncAttributeMaxDynamicSharedMemorySize,    \
                                    (int)Geo<NN>::ZSMEM));                                              \
    k_fft_z_green<NN><<<(unsigned)(batch * Geo<NN>::NCOL * (NN / Geo<NN>::TY)), Geo<NN>::ZT, Geo<NN>::ZSMEM, \
                        c->stream>>>(sp, tw, s2, del2, inv_n3);                                      \
    break;
    ZCASE(64)
    ZCASE(128)
    ZCASE(256)
    ZCASE(512)
#undef ZCASE
  }
  ktime_end(c, kt_);
  c->launches++;
  ASOHF_CUDA(cudaGetLastError());
  return ASOHF_OK;
}
