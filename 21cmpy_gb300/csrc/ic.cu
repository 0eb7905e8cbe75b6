// Initial conditions (21cmpy's Programs/initialize.py:33-111, initialize.cu:58-95, 133-190): the
// k-space pieces around the engine's inverse FFT.
//
//  * ic_spectrum: the Gaussian random field's half spectrum in numpy rfftn layout,
//    H(k) = sqrt(P(|k|) V) (n_re + i n_im) / sqrt(2) for 0 < k_z < N/2 and the Hermitian part
//    sqrt(P V) ((n_re(k) + n_re(-k)) + i (n_im(k) - n_im(-k))) / 2 on the k_z = 0 and N/2 planes, P
//    linearly interpolated in a table (init_kernel, initialize.cu:58-95).  The reference fills a
//    full complex box with independent normals and keeps the real part of its inverse FFT; that
//    real part is the inverse FFT of the Hermitian part of the box, whose modes have exactly this
//    distribution (variance P V per mode), so the half spectrum is drawn directly.
//  * ic_shape: H(k) times the smoothing window W(kR) (HII_filter, initialize.cu:12-40) and, for a
//    velocity component c, the factor i k_c / k^2 (set_velocity, initialize.cu:148-190), zero at
//    the component's Nyquist index (an odd derivative has no real value there; the reference's
//    real part drops it the same way).
//  * fold_kernel (ic_sampled_fields): ic_shape for up to four components at once, folded p-fold per axis
//    onto the spectrum of the field's every p-th cell.
//  * ic_subsample: nearest-cell subsample of a DIM^3 box onto HII_DIM^3 with a scale factor
//    (subsample, initialize.cu:133-146, and the 1 / scale^3 normalisation of initialize.py:89-109).
#include <cuda_runtime.h>
#include <stdint.h>

#include <climits>
#include <cmath>
#include <cstdarg>
#include <cstdio>
#include <string>

#include "es_engine.h"
#include "es_kernels.cuh"

namespace ic {

__device__ __forceinline__ int wrapk(int m, int n) { return m > n / 2 ? m - n : m; }

// first index i in [1, tn) with K[i] >= k (K[0] < k holds for every k > 0 of the box; tn - 1 if there is
// none): right there or one beside where a log-spaced table would have it, or else by halving what is left on that
// side.  512^3 with 4096 entries: log-spaced 233 us, linear 350 (one step after the other from the guess: 16.3 ms).
__device__ __forceinline__ int upper(const float* K, int tn, float k, float l0, float per) {
  const float g = (__log2f(k) - l0) * per + 1.0f;
  const int i = g >= 1.0f && g < (float)(tn - 1) ? (int)g : (g >= 1.0f ? tn - 1 : 1);
  int lo, hi;                                           // the index lies in (lo, hi]
  if (K[i] < k) {
    lo = i;
    hi = min(i + 1, tn - 1);
    if (K[hi] < k) { lo = hi; hi = tn - 1; }
  } else {
    hi = i;
    lo = i - 1;
    if (K[lo] >= k) { hi = max(lo, 1); lo = 0; }
  }
  while (hi - lo > 1) {
    const int mid = (lo + hi) >> 1;
    if (K[mid] >= k) hi = mid; else lo = mid;
  }
  return hi;
}

// The rows (+-k0, +-k1) of a quad: P depends on |k| alone, so what one element needs (two square roots,
// a division, the table) serves all four.  Rows at index 0 or n/2 are their own mirror images.
struct Quad {
  int rows[4], count;
  __device__ __forceinline__ Quad(int k0, int k1, int n) : count(0) {
    const bool two0 = k0 != 0 && 2 * k0 != n, two1 = k1 != 0 && 2 * k1 != n;
    rows[count++] = k0 * n + k1;
    if (two0) rows[count++] = (n - k0) * n + k1;
    if (two1) rows[count++] = k0 * n + n - k1;
    if (two0 && two1) rows[count++] = (n - k0) * n + n - k1;
  }
};

// A warp takes the row quads in turn, the table lies in shared memory (when it fits) and is entered near
// the right place: 512^3 662 us one element at a time, with a division for its index and a binary search in
// global memory, 234 us now (1.08 GB moved: 160 us).  Bound by DRAM.  With `main` it also
// writes the spectrum in a transform plan's layout, 308 us at 512^3; converting its output there took 203 us more.
constexpr int kTabMax = 2048;                         // table entries held in shared memory
__global__ void __launch_bounds__(256) spectrum_kernel(int n, float dk, const float* __restrict__ nre,
                                                       const float* __restrict__ nim, const float* __restrict__ Kg,
                                                       const float* __restrict__ Pg, int tn, float vol,
                                                       float2* __restrict__ out, float2* __restrict__ main,
                                                       float2* __restrict__ nyq) {
  __shared__ float tab[2 * kTabMax];
  const bool fits = tn <= kTabMax;
  if (fits)
    for (int i = threadIdx.x; i < tn; i += blockDim.x) { tab[i] = Kg[i]; tab[kTabMax + i] = Pg[i]; }
  __syncthreads();
  const float* K = fits ? tab : Kg;
  const float* P = fits ? tab + kTabMax : Pg;
  const float l0 = __log2f(K[0]), per = (float)(tn - 1) / (__log2f(K[tn - 1]) - l0);
  const int h = n / 2 + 1, lane = threadIdx.x & 31, step = gridDim.x * (blockDim.x / 32);
  for (int quad = blockIdx.x * (blockDim.x / 32) + (threadIdx.x >> 5); quad < h * h; quad += step) {
    const int k0 = quad / h, k1 = quad - k0 * h;        // 0 .. n/2 either
    const Quad q(k0, k1, n);
    const float kx = __fmul_rn((float)k0, dk), ky = __fmul_rn((float)k1, dk);   // the signs go with the squares
    const float kxy = __fadd_rn(__fmul_rn(kx, kx), __fmul_rn(ky, ky));
    for (int k2 = lane; k2 < h; k2 += 32) {
      const bool inner = k2 != 0 && k2 != n / 2;
      float re[4], im[4];
#pragma unroll
      for (int r = 0; r < 4; ++r) {
        if (r < q.count) {
          const size_t idx = (size_t)q.rows[r] * h + k2;
          re[r] = nre[idx];
          im[r] = nim[idx];
        }
      }
      const float kz = __fmul_rn((float)k2, dk);
      const float ksq = __fadd_rn(kxy, __fmul_rn(kz, kz));
      const float kmag = __fsqrt_rn(ksq);
      const int i = upper(K, tn, kmag, l0, per);
      // P[i-1] + (P[i] - P[i-1]) (k - K[i-1]) / (K[i] - K[i-1])   (initialize.cu:90)
      const float ps = __fadd_rn(P[i - 1], __fdiv_rn(__fmul_rn(__fsub_rn(P[i], P[i - 1]), __fsub_rn(kmag, K[i - 1])),
                                                   __fsub_rn(K[i], K[i - 1])));
      const float amp = ksq == 0.0f ? 0.0f : __fsqrt_rn(__fmul_rn(ps, vol));
      const float a = __fmul_rn(amp, 0.70710678118654752f);
#pragma unroll
      for (int r = 0; r < 4; ++r) {
        if (r < q.count) {
          const size_t idx = (size_t)q.rows[r] * h + k2;
          float2 v = make_float2(__fmul_rn(a, re[r]), __fmul_rn(a, im[r]));
          if (!inner) {
            // the k_z = 0 and N/2 planes hold both k and -k: their Hermitian part (X_k + conj X_-k) / 2,
            // real at the self-conjugate modes
            const int r0 = q.rows[r] / n, r1 = q.rows[r] % n;
            const size_t mid = ((size_t)((n - r0) % n) * n + (n - r1) % n) * h + k2;
            v = make_float2(__fmul_rn(amp, __fmul_rn(__fadd_rn(re[r], nre[mid]), 0.5f)),
                            __fmul_rn(amp, __fmul_rn(__fsub_rn(im[r], nim[mid]), 0.5f)));
          }
          if (ksq == 0.0f) v = make_float2(0.f, 0.f);
          out[idx] = v;
          if (main) (k2 < n / 2 ? main[(size_t)q.rows[r] * (n / 2) + k2] : nyq[q.rows[r]]) = v;
        }
      }
    }
  }
}

__global__ void shape_kernel(int n, float dk, const float2* __restrict__ in, int comp, int filter, float R,
                             int k2cut, int ref_compat, float2* __restrict__ out) {
  const int h = n / 2 + 1;
  const long total = (long)n * n * h;
  for (long idx = (long)blockIdx.x * blockDim.x + threadIdx.x; idx < total; idx += (long)gridDim.x * blockDim.x) {
    const int k2 = (int)(idx % h);
    const long t = idx / h;
    const int k1 = (int)(t % n), k0 = (int)(t / n);
    const int m0 = wrapk(k0, n), m1 = wrapk(k1, n);
    const int kk = m0 * m0 + m1 * m1 + k2 * k2;
    float2 v = in[idx];
    const float W = filter >= 0 ? es::filter_weight(kk, dk, R, k2cut, filter, ref_compat) : 1.0f;
    v = make_float2(v.x * W, v.y * W);
    if (comp >= 0) {
      const int mc = comp == 0 ? m0 : (comp == 1 ? m1 : k2);
      if (kk == 0 || mc == n / 2) {           // no odd derivative at the component's Nyquist index
        v = make_float2(0.f, 0.f);
      } else {
        const float kc = (float)(comp == 0 ? m0 : (comp == 1 ? m1 : k2)) * dk;
        const float f = kc / ((float)kk * dk * dk);           // k_c / k^2
        v = make_float2(-f * v.y, f * v.x);                   // i f (a + i b)
      }
    }
    out[idx] = v;
  }
}

// Keeping every p-th cell of an n^3 field (p = n / h) is folding its spectrum: with G the full shaped
// spectrum, F[k'] = sum over the aliases k = k' + m h (m < p per axis) of G[k], and the h^3 inverse
// transform of F is the sampled field.  G's upper half along the last axis is the mirror image
// conj(H[-k0, -k1, n - kz]) of the stored one.  A CTA makes the rows (+-k0', +-k1') of F for every
// component: GR groups of h/2 + 1 threads, one kz' per thread, share the p^2 aliases, an alias's window
// and 1 / k^2 serve its four sign combinations, and each element of H is read once for all components.
// 512^3 -> 128^3, four components: 247 us (0.54 GB read: 80 us; bound by latency: 285 us at 70 registers and
// three groups, 455 with the next alias' loads ahead at 90), 502 us with the window evaluated for each element; the route through ic_shape, the 512^3 inverse and ic_subsample took 1.2 ms a component.
// nyq: null for the numpy layout, else H's Nyquist plane apart.
struct FoldOut { float2 *main[4], *nyq[4]; };
template <int NC>
__global__ void __launch_bounds__(544, 2) fold_kernel(int n, int h, float dk, const float2* __restrict__ H,
                                                   const float2* __restrict__ nyq, int filter, float R, int k2cut,
                                                   int ref_compat, int first, int groups, FoldOut o) {
  extern __shared__ float2 part[];                      // [groups][4][NC][h/2 + 1]
  const int w = h / 2 + 1, p = n / h, m = n / 2;
  const int kp = threadIdx.x % w, gr = threadIdx.x / w;
  const int r0 = blockIdx.x / w, r1 = blockIdx.x % w;   // 0 .. h/2 either
  const bool two0 = r0 != 0 && 2 * r0 != h, two1 = r1 != 0 && 2 * r1 != h;   // rows that are not their own mirror image
  float2 acc[4][NC];
#pragma unroll
  for (int s = 0; s < 4; ++s)
#pragma unroll
    for (int c = 0; c < NC; ++c) acc[s][c] = make_float2(0.f, 0.f);
  if (gr < groups) {
    // the mode itself (q = 0, mz = 0) last: it is the largest of its aliases as a rule, and sums that end
    // with it round once at its size instead of p^3 times
    for (int q = gr + (p * p - 1 - gr) / groups * groups; q >= 0; q -= groups) {
      const int k0 = r0 + (q / p) * h, k1 = r1 + (q % p) * h;
      const int m0 = wrapk(k0, n), m1 = wrapk(k1, n);
      const int n0 = k0 ? n - k0 : 0, n1 = k1 ? n - k1 : 0;
      for (int mz = p - 1; mz >= 0; --mz) {
        const int kz = kp + mz * h;
        const bool up = kz > m;
        const int z = up ? n - kz : kz;                 // stored column
        const int kk = m0 * m0 + m1 * m1 + z * z;
        float2 v[4];
#pragma unroll
        for (int s = 0; s < 4; ++s) {
          if ((!(s & 1) || two0) && (!(s & 2) || two1)) {
            // combination s: k0 negated by bit 0, k1 by bit 1; an upper element is stored at -k
            const int a0 = ((s & 1) != 0) != up ? n0 : k0, a1 = ((s & 2) != 0) != up ? n1 : k1;
            const size_t row = (size_t)a0 * n + a1;
            v[s] = nyq ? (z < m ? H[row * m + z] : nyq[row]) : H[row * (m + 1) + z];
          } else {
            v[s] = make_float2(0.f, 0.f);
          }
        }
        const float W = filter >= 0 ? es::filter_weight(kk, dk, R, k2cut, filter, ref_compat) : 1.0f;
        const float inv = kk ? 1.0f / ((float)kk * dk) : 0.f;     // k_c / k^2 = m_c / (|m|^2 dk)
        // no odd derivative at the Nyquist index
        const float f0 = m0 == m ? 0.f : (float)m0 * inv, f1 = m1 == m ? 0.f : (float)m1 * inv;
        const float f2 = z == m ? 0.f : (float)(up ? -z : z) * inv;
#pragma unroll
        for (int s = 0; s < 4; ++s) {
          const float x = v[s].x * W, y = up ? -v[s].y * W : v[s].y * W;
#pragma unroll
          for (int c = 0; c < NC; ++c) {
            const int comp = first + c;
            if (comp < 0) {                             // the product unrounded: x is rounded for the other components
              acc[s][c].x = fmaf(v[s].x, W, acc[s][c].x);
              acc[s][c].y = fmaf(up ? -v[s].y : v[s].y, W, acc[s][c].y);
            } else {
              const float f = comp == 0 ? (s & 1 ? -f0 : f0) : comp == 1 ? (s & 2 ? -f1 : f1) : f2;
              acc[s][c].x -= f * y;
              acc[s][c].y += f * x;
            }
          }
        }
      }
    }
  }
  auto row_of = [&](int s) { return (s & 1 ? h - r0 : r0) * h + (s & 2 ? h - r1 : r1); };
  auto put = [&](int s, int c, int k, float2 v) {
    if ((!(s & 1) || two0) && (!(s & 2) || two1)) {
      if (k < h / 2) o.main[c][(size_t)row_of(s) * (h / 2) + k] = v;
      else o.nyq[c][row_of(s)] = v;
    }
  };
  if (groups == 1) {
    if (gr == 0) {
#pragma unroll
      for (int s = 0; s < 4; ++s)
#pragma unroll
        for (int c = 0; c < NC; ++c) put(s, c, kp, acc[s][c]);
    }
    return;
  }
  if (gr < groups) {
#pragma unroll
    for (int s = 0; s < 4; ++s)
#pragma unroll
      for (int c = 0; c < NC; ++c) part[((gr * 4 + s) * NC + c) * w + kp] = acc[s][c];
  }
  __syncthreads();
  for (int i = threadIdx.x; i < 4 * NC * w; i += blockDim.x) {
    float2 t = make_float2(0.f, 0.f);
    for (int g = groups - 1; g >= 0; --g) {
      const float2 v = part[g * 4 * NC * w + i];
      t.x += v.x;
      t.y += v.y;
    }
    put(i / (NC * w), (i / w) % NC, i % w, t);
  }
}

__global__ void subsample_kernel(int dim, int sw, float pf, float scale, const float* __restrict__ large,
                                 float* __restrict__ small) {
  const long total = (long)sw * sw * sw;
  for (long idx = (long)blockIdx.x * blockDim.x + threadIdx.x; idx < total; idx += (long)gridDim.x * blockDim.x) {
    const int a2 = (int)(idx % sw);
    const long t = idx / sw;
    const int a1 = (int)(t % sw), a0 = (int)(t / sw);
    int l[3];
    const int a[3] = {a0, a1, a2};
#pragma unroll
    for (int d = 0; d < 3; ++d) {
      int li = (int)floorf(__fadd_rn(__fmul_rn((float)a[d], pf), 0.5f));
      l[d] = li < 0 ? 0 : (li >= dim ? dim - 1 : li);
    }
    small[idx] = __fmul_rn(large[((size_t)l[0] * dim + l[1]) * dim + l[2]], scale);
  }
}

}  // namespace ic

namespace {
thread_local std::string g_ic_error;
int icfail(int code, const char* fmt, ...) {
  char buf[512];
  va_list ap;
  va_start(ap, fmt);
  vsnprintf(buf, sizeof(buf), fmt, ap);
  va_end(ap);
  g_ic_error = buf;
  return code;
}
unsigned grid_for(long total) {
  int dev = 0, sms = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  long b = (total + 255) / 256;
  const long cap = (long)sms * 8;
  return (unsigned)(b < 1 ? 1 : (b > cap ? cap : b));
}
}  // namespace

// k-space top-hat keeps modes with (dk |k| R) 0.413566994 <= 1 (initialize.cu:31-34)
static int tophat_cut(float dk, int filter_type, float R, int ref_compat) {
  if (!(filter_type == 1 || (ref_compat && filter_type == 0))) return INT_MAX;
  const double d = dk, r = R;
  long m = (long)std::floor(std::pow(1.0 / (0.413566994 * d * r), 2)) + 2;
  while (m >= 0 && (d * std::sqrt((double)m) * r) * 0.413566994 > 1.0) --m;
  return (int)(m < (long)INT_MAX ? m : (long)INT_MAX);
}

__attribute__((visibility("hidden"))) cudaError_t ic_launch_fold(int n, int h, float dk, const float2* half, const float2* nyq, int filter, float R, int ref_compat,
                           int first, int count, float2* const* out, float2* const* out_nyq, cudaStream_t s) {
  const int w = h / 2 + 1;
  // up to 288 threads, and of those the fewest groups that take the alias rows in as many rounds: at
  // 512 -> 128 four groups take 16 rows in 4 (three in 6: 266 us against 285).  Rows of more than 96 values keep
  // to 256 threads: their few aliases (p = 2) are better added up by one group, error against float64 2.22e-7
  // of a 512 -> 256 velocity box against 2.27e-7 by two
  const int p2 = (n / h) * (n / h), fit = (w <= 96 ? 288 : 256) / w, most = fit < 1 ? 1 : (fit > p2 ? p2 : fit);
  const int rounds = (p2 + most - 1) / most, groups = (p2 + rounds - 1) / rounds;
  const int threads = (groups * w + 31) / 32 * 32;
  const size_t smem = groups > 1 ? (size_t)groups * 4 * count * w * sizeof(float2) : 0;   // at most 36 KB
  const int cut = tophat_cut(dk, filter, R, ref_compat);
  ic::FoldOut o{};
  for (int i = 0; i < count; ++i) { o.main[i] = out[i]; o.nyq[i] = out_nyq[i]; }
#define IC_FOLD(NC)                                                                                                   \
  case NC:                                                                                                            \
    ic::fold_kernel<NC><<<w * w, threads, smem, s>>>(n, h, dk, half, nyq, filter, R, cut, ref_compat, first, groups, o); \
    break
  switch (count) {
    IC_FOLD(1);
    IC_FOLD(2);
    IC_FOLD(3);
    IC_FOLD(4);
    default: return cudaErrorInvalidValue;
  }
#undef IC_FOLD
  return cudaGetLastError();
}

// es_engine.cu: the spectrum in numpy's layout and, if main is given, in a transform plan's
__attribute__((visibility("hidden"))) cudaError_t ic_launch_spectrum(int n, float box_len, const float* nre, const float* nim, const float* K,
                               const float* P, int tn, float2* out, float2* main, float2* nyq, cudaStream_t s) {
  const float dk = (float)(2.0 * M_PI / (double)box_len);
  const float vol = box_len * box_len * box_len;
  ic::spectrum_kernel<<<grid_for((long)n * n * (n / 2 + 1)), 256, 0, s>>>(n, dk, nre, nim, K, P, tn, vol, out, main, nyq);
  return cudaGetLastError();
}

extern "C" {

int ic_spectrum(int n, float box_len, const float* normals_re, const float* normals_im, const float* k_table,
                const float* p_table, int table_n, void* out_half, void* stream) {
  if (n < 2 || n > 2048 || !(box_len > 0.f) || !normals_re || !normals_im || !k_table || !p_table || !out_half ||
      table_n < 2)
    return icfail(ES_E_ARG, "ic_spectrum: bad arguments");
  const cudaError_t e = ic_launch_spectrum(n, box_len, normals_re, normals_im, k_table, p_table, table_n, (float2*)out_half,
                                           nullptr, nullptr, (cudaStream_t)stream);
  return e == cudaSuccess ? ES_OK : icfail(ES_E_CUDA, "ic_spectrum launch: %s", cudaGetErrorString(e));
}

int ic_shape(int n, float box_len, const void* in_half, int component, int filter_type, float R, int ref_compat,
             void* out_half, void* stream) {
  if (n < 2 || n > 2048 || !(box_len > 0.f) || !in_half || !out_half || component < -1 || component > 2 ||
      filter_type < -1 || filter_type > 2)
    return icfail(ES_E_ARG, "ic_shape: bad arguments");
  const float dk = (float)(2.0 * M_PI / (double)box_len);
  const int k2cut = tophat_cut(dk, filter_type, R, ref_compat);
  const long total = (long)n * n * (n / 2 + 1);
  ic::shape_kernel<<<grid_for(total), 256, 0, (cudaStream_t)stream>>>(n, dk, (const float2*)in_half, component,
                                                                       filter_type, R, k2cut, ref_compat,
                                                                       (float2*)out_half);
  const cudaError_t e = cudaGetLastError();
  return e == cudaSuccess ? ES_OK : icfail(ES_E_CUDA, "ic_shape launch: %s", cudaGetErrorString(e));
}

int ic_subsample(int dim, int hii_dim, float pixel_factor, float scale, const float* large, float* small,
                 void* stream) {
  if (dim < 1 || hii_dim < 1 || hii_dim > dim || !(pixel_factor > 0.f) || !large || !small)
    return icfail(ES_E_ARG, "ic_subsample: bad arguments");
  const long total = (long)hii_dim * hii_dim * hii_dim;
  ic::subsample_kernel<<<grid_for(total), 256, 0, (cudaStream_t)stream>>>(dim, hii_dim, pixel_factor, scale, large,
                                                                           small);
  const cudaError_t e = cudaGetLastError();
  return e == cudaSuccess ? ES_OK : icfail(ES_E_CUDA, "ic_subsample launch: %s", cudaGetErrorString(e));
}

int ic_last_error(char* buf, int len) {
  if (!buf || len <= 0) return ES_E_ARG;
  std::snprintf(buf, (size_t)len, "%s", g_ic_error.c_str());
  return ES_OK;
}

}  // extern "C"
