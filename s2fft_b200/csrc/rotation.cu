// Rotation of spherical-harmonic coefficients by Euler angles (alpha, beta, gamma):
//   flm'[l, m] = exp(-i m alpha) sum_n d^l_{m,n}(beta) exp(-i n gamma) flm[l, n]
// (upstream s2fft/utils/rotation.py:9-64, rotate_flms; the planes of generate_rotate_dls,
// rotation.py:75-96).
//
// Upstream builds the Wigner-d planes degree by degree with Risbo's recursion
// (s2fft/recursions/risbo.py:4-120), so every degree waits for the whole previous plane.
// Here each (l, m) walks along n by its own three-term recurrence, fused with the sum over n
// (rotate_walk_kernel). All arithmetic is double.
//
// The planes (generate_rotate_dls) are written once per entry, so there every (m, n) follows
// its three-term recurrence in the degree, whose stores are consecutive in n
// (Varshalovich, Moskalev & Khersonskii, Quantum Theory of Angular Momentum, sec. 4.8;
// Kostelec & Rockmore, J. Fourier Anal. Appl. 14 (2008) 145-179):
//   d^{l+1}_{mn} = U_l(m) R_l(n) [ (cos beta - m n q_l) d^l_{mn} - V_l(m) P_l(n) d^{l-1}_{mn} ],
//   R_l(k) = 1/sqrt((l+1)^2 - k^2), P_l(k) = sqrt(l^2 - k^2), q_l = 1/(l(l+1)),
//   U_l(m) = (l+1)(2l+1) R_l(m), V_l(m) = P_l(m) / (l(2l+1)),
// started at l0 = max(|m|, |n|) from E[l0][a] = d^{l0}_{l0,a} = (-1)^{l0-a}
// sqrt(binom(2 l0, l0+a)) c^{l0+a} s^{l0-a} (c = cos(beta/2), s = sin(beta/2)) through
// d_{m,n} = (-1)^{m-n} d_{n,m} = d_{-n,-m}. Orders m < 0 follow from
// d_{-m,-n} = (-1)^{m-n} d_{m,n}, so only m >= 0 is recurred.
//
// Start values below 2^-960 are carried there as a mantissa times 2^k (an int k < 0 per
// entry), renormalised in steps of 2^64 as they grow, and weighted by 2^k where they
// contribute. The start table is the exponent-tracked product W = E^2,
//   W_l = W_{l-1} 2l(2l-1) / ((l+a)(l-a)) (cs)^2,  W_{|a|} = c^{4a} (a >= 0), s^{4|a|} (a < 0),
// formed in segments of 32 degrees with a carry pass, so no log-gamma enters.
// A lane carries MT x S recurrences (MT orders, S values of n) in registers and walks l from
// m0 to L-1; its operand T[l][|n|] arrives through a cp.async ring in shared memory a few
// degrees ahead. Every entry of [L][2L-1][2L-1] is written once, zeros included.
#include <cuda_runtime.h>
#include <math_constants.h>

#include <cmath>
#include <cstdint>
#include <type_traits>
#include <utility>

#include "s2b.h"
#include "s2b_dev.h"
#include "s2b_internal.h"
#include "s2b_rotation.h"

namespace s2b {
namespace {

constexpr int kRotSeg = 32;    // degrees per segment of the start-table product
constexpr int kRotChunk = 16;  // degrees of a staged coefficient chunk

template <typename R2>
struct RotIO;
template <>
struct RotIO<float2> {
  static __device__ double2 get(const void* p, size_t i) {
    const float2 v = __ldg(reinterpret_cast<const float2*>(p) + i);
    return make_double2(v.x, v.y);
  }
  static __device__ void put(void* p, size_t i, double2 v) {
    reinterpret_cast<float2*>(p)[i] = make_float2((float)v.x, (float)v.y);
  }
};
template <>
struct RotIO<double2> {
  static __device__ double2 get(const void* p, size_t i) {
    return __ldg(reinterpret_cast<const double2*>(p) + i);
  }
  static __device__ void put(void* p, size_t i, double2 v) {
    reinterpret_cast<double2*>(p)[i] = v;
  }
};

__device__ __forceinline__ double warp_sum(double v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// ---------------------------------------------------------------------------------
// tables
// ---------------------------------------------------------------------------------

// recurrence coefficients T and UVQ (beta-independent)
__global__ void rotate_coef_kernel(RotParams p) {
  const int L = p.L;
  const long total = (long)L * L;
  for (long e = blockIdx.x * (long)blockDim.x + threadIdx.x; e < total;
       e += (long)gridDim.x * blockDim.x) {
    const int l = (int)(e / L), k = (int)(e % L);
    double2 t = make_double2(0.0, 0.0);
    double4 uv = make_double4(0.0, 0.0, 0.0, 0.0);
    if (k <= l) {
      const double dl = (double)l, dk = (double)k;
      const double R = 1.0 / sqrt((dl + 1.0) * (dl + 1.0) - dk * dk);
      const double P = sqrt(dl * dl - dk * dk);
      t = make_double2(R, P);
      if (l > 0)
        uv = make_double4((dl + 1.0) * (2.0 * dl + 1.0) * R, P / (dl * (2.0 * dl + 1.0)),
                          -dk / (dl * (dl + 1.0)), 0.0);
      else
        uv = make_double4(R, 0.0, 0.0, 0.0);
    }
    p.T[e] = t;
    p.UVQ[e] = uv;
  }
}

__device__ __forceinline__ RotXD xd_make(double x) {
  RotXD r;
  r.m = frexp(x, &r.e);
  r.pad = 0;
  if (r.m == 0.0) r.e = 0;
  return r;
}
__device__ __forceinline__ RotXD xd_mul(RotXD a, RotXD b) {
  int d;
  RotXD r;
  r.m = frexp(a.m * b.m, &d);
  r.e = r.m == 0.0 ? 0 : a.e + b.e + d;
  r.pad = 0;
  return r;
}
__device__ RotXD xd_pow(double x, int n) {  // x^n, n >= 0
  RotXD r = xd_make(1.0), b = xd_make(x);
  while (n) {
    if (n & 1) r = xd_mul(r, b);
    b = xd_mul(b, b);
    n >>= 1;
  }
  return r;
}

// start table, pass 1: W_l / W_{segment start} inside each segment of kRotSeg degrees
// (the segment holding l = |a| starts from W_{|a|}); the segment product goes to carry
__global__ void rotate_start_seg_kernel(RotParams p) {
  const int L = p.L, NN = 2 * L - 1;
  const int ai = blockIdx.x * blockDim.x + threadIdx.x, g = blockIdx.y;
  if (ai >= NN) return;
  const int a = ai - (L - 1), aa = a < 0 ? -a : a;
  const int lb = max(g * kRotSeg, aa), le = min(g * kRotSeg + kRotSeg, L);
  RotXD w = xd_make(1.0);
  if (lb < le) {
    if (lb == aa) w = a >= 0 ? xd_pow(p.c2, 2 * a) : xd_pow(p.s2, 2 * aa);
#pragma unroll 1
    for (int l = lb; l < le; ++l) {
      if (l > aa) {
        const double f = (2.0 * l) * (2.0 * l - 1.0) / ((double)(l + a) * (double)(l - a));
        w = xd_mul(w, xd_make(f * p.cs2));
      }
      p.start[(size_t)l * NN + ai] = w;
    }
  }
  p.carry[(size_t)g * NN + ai] = w;
}

// pass 2: exclusive products of the segment products, per a
__global__ void rotate_start_carry_kernel(RotParams p) {
  const int L = p.L, NN = 2 * L - 1, G = (L + kRotSeg - 1) / kRotSeg;
  const int ai = blockIdx.x * blockDim.x + threadIdx.x;
  if (ai >= NN) return;
  RotXD c = xd_make(1.0);
#pragma unroll 1
  for (int g0 = 0; g0 < G; g0 += 8) {  // eight segment products in flight at a time
    RotXD t[8];
#pragma unroll
    for (int u = 0; u < 8; ++u)
      if (g0 + u < G) t[u] = p.carry[(size_t)(g0 + u) * NN + ai];
#pragma unroll
    for (int u = 0; u < 8; ++u)
      if (g0 + u < G) {
        p.carry[(size_t)(g0 + u) * NN + ai] = c;
        c = xd_mul(c, t[u]);
      }
  }
}

// pass 3: E = sign sqrt(W) as the start value (v, k) of the recurrence
__global__ void rotate_start_final_kernel(RotParams p) {
  const int L = p.L, NN = 2 * L - 1;
  const int ai = blockIdx.x * blockDim.x + threadIdx.x, l = blockIdx.y;
  if (ai >= NN) return;
  const int a = ai - (L - 1);
  if (a < -l || a > l) return;
  const size_t e = (size_t)l * NN + ai;
  const RotXD w = xd_mul(p.start[e], p.carry[(size_t)(l / kRotSeg) * NN + ai]);
  double m = w.m;
  int x = w.e;
  if (x & 1) {
    m *= 2.0;
    x -= 1;
  }
  RotXD r;
  r.pad = 0;
  r.m = sqrt(m);
  r.e = x / 2;
  if (m == 0.0) {
    r.e = 0;
  } else if (r.e >= -960) {
    r.m = ldexp(r.m, r.e);
    r.e = 0;
  }
  const int neg = ((l - a) & 1) ^ (p.c_neg & ((l + a) & 1)) ^ (p.s_neg & ((l - a) & 1));
  if (neg) r.m = -r.m;
  p.start[e] = r;
}

// ---------------------------------------------------------------------------------
// recurrence kernel
// ---------------------------------------------------------------------------------

// 2^k for -1022 <= k <= 0, 0 below (a term of at most 2^(64+k) is then far below rounding)
__device__ __forceinline__ double pow2k(int k) {
  return k < -1022 ? 0.0 : __hiloint2double((k + 1023) << 20, 0);
}

// coefficients UVQ[l][m0 + i] of kRotChunk degrees from l0 into uvq[lc][i] (cp.async)
template <int MT>
__device__ __forceinline__ void rotate_stage(const RotParams& p, double4* uvq, int l0, int m0) {
  for (int e = threadIdx.x; e < 2 * kRotChunk * MT; e += blockDim.x) {
    const int h = e & 1, lc = (e >> 1) / MT, i = (e >> 1) % MT, l = l0 + lc;
    const double4* src = p.UVQ + (size_t)min(l, p.L - 1) * p.L + min(m0 + i, p.L - 1);
    cp_async<16>((unsigned)__cvta_generic_to_shared(uvq + lc * MT + i) + 16 * h,
                 reinterpret_cast<const char*>(src) + 16 * h, l < p.L);
  }
}

template <int S>
constexpr int rot_depth() {  // degrees of the per-lane copy pipeline
  return S == 1 ? 4 : S == 2 ? 3 : 2;
}

// The planes kernel. p.nr CTAs (rank blockIdx.x) own the orders m0 = MT blockIdx.y ..
// m0 + MT - 1. Dynamic shared memory:
//   ring  [D][S][blockDim] double2: T[l][|n|] of each lane, copied D - 1 degrees ahead
//   uvq   [2][kRotChunk][MT] double4 coefficients, staged a chunk ahead
template <int MT, int S>
__global__ void __launch_bounds__(kRotThreads, 2) rotate_lrec_kernel(RotParams p) {
  extern __shared__ double4 smem4[];
  constexpr int D = rot_depth<S>();
  static_assert(MT % 2 == 0, "tiles start at even orders");
  const int L = p.L, NN = 2 * L - 1;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, nt = blockDim.x;
  const int nw = p.nw, nr = p.nr, rank = blockIdx.x;
  const int m0 = blockIdx.y * MT;
  double* const dl = p.dl_out;
  double2* const ring = reinterpret_cast<double2*>(smem4);
  double4* const uvq = smem4 + (D * S * nt) / 2;

  // this lane's n, one per S, in natural order (j -> j - (L-1)), so that a warp's stores
  // cover 32 consecutive columns
  int nv[S], an[S], wmin[S], wmax[S];
  double nd[S];
#pragma unroll
  for (int s = 0; s < S; ++s) {
    const int gw = (s * nw + warp) * nr + rank;  // warp slot in the order of n
    const int j = gw * 32 + lane;
    const bool ok = j < NN;
    nv[s] = ok ? j - (L - 1) : 0;
    nd[s] = (double)nv[s];
    an[s] = ok ? abs(nv[s]) : L;  // L: never starts
    // least and largest |n| of the warp slot's (valid) n
    const int lo = gw * 32 - (L - 1), hi = min(lo + 31, L - 1);
    wmin[s] = (lo <= 0 && hi >= 0) ? 0 : min(abs(lo), abs(hi));
    wmax[s] = max(abs(lo), abs(hi));
  }
  // degrees at which some entry of the warp slot starts: max(m, |n|) over its orders and lanes
  int wlo[S], whi[S], wany = wmin[0];  // wany: least |n| of the warp
#pragma unroll
  for (int s = 0; s < S; ++s) {
    wlo[s] = max(m0, wmin[s]);
    whi[s] = min(L - 1, max(m0 + MT - 1, wmax[s]));
    wany = min(wany, wmin[s]);
  }

  // degrees below m0: the tile's rows are zero there
#pragma unroll 1
  for (int l = 0; l < m0; ++l)
#pragma unroll
    for (int s = 0; s < S; ++s) {
      if (an[s] >= L) continue;
#pragma unroll
      for (int i = 0; i < MT; ++i) {
        const int m = m0 + i;
        if (m >= L) continue;
        dl[((size_t)l * NN + L - 1 + m) * NN + L - 1 + nv[s]] = 0.0;
        if (m > 0) dl[((size_t)l * NN + L - 1 - m) * NN + L - 1 - nv[s]] = 0.0;
      }
    }
  // copies of consecutive degrees ll = m0, m0 + 1, ... into ring stage st (zero where
  // nothing has started); with one n per lane the source pointer advances by one row
  // per call, with more they are recomputed (fewer live registers)
  const unsigned rbase = (unsigned)__cvta_generic_to_shared(ring + tid);
  const double2* tq = p.T + (size_t)m0 * L + min(an[0], L - 1);
  int ll = m0;
  auto issue = [&](int st) {
#pragma unroll
    for (int s = 0; s < S; ++s) {
      const bool vt = ll < L && ll >= wmin[s];
      const int lt = min(ll, L - 1);
      const double2* ts = S == 1 ? tq : p.T + (size_t)lt * L + min(an[s], L - 1);
      cp_async<16>(rbase + (unsigned)((st * S + s) * nt) * 16u, ts, vt);
    }
    if (S == 1 && ll + 1 < L) tq += L;
    ++ll;
  };
  rotate_stage<MT>(p, uvq, m0, m0);
  cp_async_commit();
#pragma unroll
  for (int k = 0; k < D - 1; ++k) {
    issue(k);
    cp_async_commit();
  }
  cp_async_wait<D - 1>();  // the coefficients of the first chunk
  __syncthreads();

  double v[MT][S], vp[MT][S];
  int kx[MT][S];
#pragma unroll
  for (int i = 0; i < MT; ++i)
#pragma unroll
    for (int s = 0; s < S; ++s) {
      v[i][s] = 0.0;
      vp[i][s] = 0.0;
      kx[i][s] = 0;
    }
  // some lane of the warp carries a start value below 2^-960 (kx < 0): warp-uniform
  bool scaled = false;
  int lc = 0, ub = 0, rs = 0;  // degree in chunk, coefficient buffer, ring stage
#pragma unroll 1
  for (int l = m0; l < L; ++l) {
    const bool step = l + 1 < L;
    // copies D - 1 degrees ahead, and the next chunk's coefficients at a chunk start
    issue(rs == 0 ? D - 1 : rs - 1);  // degree l + D - 1
    if (lc == 0 && l + kRotChunk < L)
      rotate_stage<MT>(p, uvq + (ub ^ 1) * kRotChunk * MT, l + kRotChunk, m0);
    cp_async_commit();
    cp_async_wait<D - 1>();  // this degree's copies (this thread's own)
    double2 tn[S];
#pragma unroll
    for (int s = 0; s < S; ++s) tn[s] = ring[(rs * S + s) * nt + tid];
    rs = rs == D - 1 ? 0 : rs + 1;
    const double4* const uvl = uvq + (ub * kRotChunk + lc) * MT;

    // entries starting at this degree (only inside the warp slot's start window)
#pragma unroll
    for (int s = 0; s < S; ++s) {
      if (l < wlo[s] || l > whi[s]) continue;
      bool neg = false;
#pragma unroll
      for (int i = 0; i < MT; ++i) {
        const int m = m0 + i;
        if (l == max(m, an[s])) {  // E[l][col] (symmetries of d)
          int col;
          bool flip = false;
          if (m >= an[s]) {
            col = nv[s];
          } else if (nv[s] > 0) {
            col = m;
            flip = ((m - nv[s]) & 1) != 0;
          } else {
            col = -m;
          }
          const RotXD e0 = p.start[(size_t)l * NN + L - 1 + col];
          v[i][s] = flip ? -e0.m : e0.m;
          kx[i][s] = e0.e;
          vp[i][s] = 0.0;
        }
        neg |= kx[i][s] < 0;
      }
      scaled = __any_sync(0xffffffffu, neg) || scaled;
    }
    // warp slots not started yet: their entries of the planes are 0
#pragma unroll
    for (int s = 0; s < S; ++s) {
      if (l >= wmin[s] || an[s] >= L) continue;
#pragma unroll
      for (int i = 0; i < MT; ++i) {
        const int m = m0 + i;
        if (m >= L) continue;
        dl[((size_t)l * NN + L - 1 + m) * NN + L - 1 + nv[s]] = 0.0;
        if (m > 0) dl[((size_t)l * NN + L - 1 - m) * NN + L - 1 - nv[s]] = 0.0;
      }
    }

    // one degree of every started entry, branch-free so that the MT x S recurrences
    // interleave; SC: with the 2^kx weights and the renormalisation
    auto advance = [&](auto sc_tag) {
      constexpr bool SC = decltype(sc_tag)::value;
#pragma unroll
      for (int i = 0; i < MT; ++i) {
        const double4 uv = uvl[i];
#pragma unroll
        for (int s = 0; s < S; ++s) {
          if (S > 1 && l < wmin[s]) continue;  // warp-uniform
          double dv = v[i][s];
          if constexpr (SC) dv *= pow2k(kx[i][s]);
          const int m = m0 + i;
          if (an[s] < L && m < L) {
            dl[((size_t)l * NN + L - 1 + m) * NN + L - 1 + nv[s]] = dv;
            if (m > 0)
              dl[((size_t)l * NN + L - 1 - m) * NN + L - 1 - nv[s]] =
                  ((m - nv[s]) & 1) ? -dv : dv;
          }
          if (step) {
            const double t = fma(uv.z, nd[s], p.cb);
            double vn = (uv.x * tn[s].x) * fma(t, v[i][s], -(uv.y * tn[s].y) * vp[i][s]);
            double vc = v[i][s];
            if constexpr (SC) {  // renormalise by up to 2^64 once |vn| >= 2^65
              const bool big =
                  kx[i][s] < 0 && (__double2hiint(vn) & 0x7ff00000) > ((1023 + 64) << 20);
              const int sh = big ? min(64, -kx[i][s]) : 0;
              const double f = __hiloint2double((1023 - sh) << 20, 0);
              vn *= f;
              vc *= f;
              kx[i][s] += sh;
            }
            vp[i][s] = vc;
            v[i][s] = vn;
          }
        }
      }
      if constexpr (SC) {
        bool neg = false;
#pragma unroll
        for (int i = 0; i < MT; ++i)
#pragma unroll
          for (int s = 0; s < S; ++s) neg |= kx[i][s] < 0;
        scaled = __any_sync(0xffffffffu, neg);
      }
    };
    if (l >= wany) {  // some entry of the warp has started (warp-uniform)
      if (scaled)
        advance(std::true_type{});
      else
        advance(std::false_type{});
    }

    if (lc == kRotChunk - 1 || l == L - 1) {
      __syncthreads();  // the next chunk's coefficients in place
      ub ^= 1;
      lc = 0;
    } else {
      ++lc;
    }
  }
  cp_async_wait<0>();  // the pipeline's trailing (empty) copies
}

// ---------------------------------------------------------------------------------
// rotation: the walk along n
// ---------------------------------------------------------------------------------

// a + b = hi + lo (|hi| >= |lo|), with a binary exponent: the running products of the tables
struct DDX {
  double h, l;
  int e;
};
__device__ __forceinline__ DDX ddx_mul(DDX a, DDX b) {
  const double p = a.h * b.h;
  const double r = fma(a.h, b.h, -p) + fma(a.h, b.l, a.l * b.h);
  const double h = p + r, l = r - (h - p);
  int d;
  DDX o;
  o.h = frexp(h, &d);
  if (o.h == 0.0) d = 0;
  o.l = ldexp(l, -d);
  o.e = a.e + b.e + d;
  return o;
}
__device__ DDX ddx_pow(DDX b, int n) {  // b^n, n >= 0
  DDX r{0.5, 0.0, 1};
  while (n) {
    if (n & 1) r = ddx_mul(r, b);
    b = ddx_mul(b, b);
    n >>= 1;
  }
  return r;
}
// the square root of a (a >= 0), as mantissa and exponent
__device__ __forceinline__ RotXD ddx_sqrt(DDX a) {
  if (a.e & 1) {
    a.h *= 2.0;
    a.l *= 2.0;
    a.e -= 1;
  }
  RotXD r;
  const double q = sqrt(a.h);
  r.m = q > 0.0 ? q + (fma(-q, q, a.h) + a.l) / (2.0 * q) : 0.0;
  r.e = a.e / 2;
  r.pad = 0;
  return r;
}

// W(j) = Gamma((j+1)/2) / (sqrt(pi) Gamma(j/2 + 1)): W(0) = 1, W(1) = 2/pi,
// W(j) = W(j-2) (j-1)/j; from j = 32 the expansion of the logarithm of the gamma ratio in
// 1/j (Bernoulli numbers), whose first omitted term is below 1e-17 there
__device__ double rot_w(int j) {
  if (j < 32) {
    double w = (j & 1) ? 0.63661977236758134308 : 1.0;
    for (int k = 2 + (j & 1); k <= j; k += 2) w = w * (double)(k - 1) / (double)k;
    return w;
  }
  const double z = 0.5 * (double)j, i = 1.0 / z, i2 = i * i;
  double s = 691.0 / 180224.0;
  s = fma(s, i2, -31.0 / 18432.0);
  s = fma(s, i2, 17.0 / 14336.0);
  s = fma(s, i2, -1.0 / 640.0);
  s = fma(s, i2, 1.0 / 192.0);
  s = fma(s, i2, -1.0 / 8.0);
  return exp(s * i) / sqrt(3.14159265358979323846 * z);
}

// Tables of one rotation (each of at most 2L entries): the phases, W, the powers of
// cos(beta/2) and sin(beta/2), and (the last CTA) sqrt(k!), a scan of double-double products
// so that the start values carry a few roundings only. With caller planes: the phases alone.
constexpr int kRotTab = 1024;
__global__ void __launch_bounds__(kRotTab) rotate_tables_kernel(RotParams p) {
  const int L = p.L, NN = 2 * L - 1, tid = threadIdx.x;
  if (!p.dl_in && blockIdx.x == gridDim.x - 1) {
    __shared__ DDX tot[2][kRotTab];
    const int per = (2 * L + kRotTab - 1) / kRotTab, k0 = tid * per;
    DDX a{0.5, 0.0, 1};
    auto times = [](DDX x, int k) {
      int d;
      DDX f{0.0, 0.0, 0};
      f.h = frexp((double)(k > 0 ? k : 1), &d);
      f.e = d;
      return ddx_mul(x, f);
    };
    for (int k = k0; k < min(k0 + per, 2 * L); ++k) a = times(a, k);
    int cur = 0;
    tot[0][tid] = a;
    __syncthreads();
    for (int o = 1; o < kRotTab; o <<= 1) {
      DDX t = tot[cur][tid];
      if (tid >= o) t = ddx_mul(t, tot[cur][tid - o]);
      tot[cur ^ 1][tid] = t;
      cur ^= 1;
      __syncthreads();
    }
    a = tid ? tot[cur][tid - 1] : DDX{0.5, 0.0, 1};
    for (int k = k0; k < min(k0 + per, 2 * L); ++k) {
      a = times(a, k);
      p.sqf[k] = ddx_sqrt(a);
    }
    return;
  }
  const int i = blockIdx.x * kRotTab + tid;
  if (i < NN) {
    const double k = (double)(i - (L - 1));
    double s, c;
    sincos(-k * p.alpha, &s, &c);
    p.ea[i] = make_double2(c, s);
    sincos(-k * p.gamma, &s, &c);
    p.eg[i] = make_double2(c, s);
  }
  if (!p.dl_in && i < 2 * L) {
    p.w[i] = rot_w(i);
    auto power = [i](double h, double l) {
      int d;
      DDX b;
      b.h = frexp(h, &d);
      b.l = ldexp(l, -d);
      b.e = d;
      const DDX r = ddx_pow(b, i);
      RotXD o;
      o.m = r.h + r.l;
      o.e = r.e;
      o.pad = 0;
      return o;
    };
    p.cpow[i] = power(p.ch, p.cl);
    p.spow[i] = power(p.sh, p.sl);
  }
}

constexpr int kWalkThreads = 128;  // also the steps of a staged chunk

// The rotation. For fixed (l, m) the values along n obey
//   a_n d_{m,n-1} + a_{n+1} d_{m,n+1} = 2 (n cos b - m)/sin b d_{m,n},
//   a_n = sqrt((l+n)(l-n+1)),
// and with d_{m,n} = g_n x_n, g_n^2 = W(l-n) W(l+n), the step is monic:
//   x_{n-1} = -t x_n - x_{n+1},   t = A_n (m - n) + C_n,
//   A_n = pi W(l-n) W(l+n) / sin b,   C_n = A_n n (1 - cos b).
// A lane owns orders m of one degree l and walks n downwards, so the sum over n stays in its
// registers and A, C and the weights g_n e^{-in gamma} flm[l, +-n] are warp-wide broadcasts:
// two FP64 operations for a value and four for its products with flm[n] (order m) and, by
// d_{-m,-n} = (-1)^{m-n} d_{m,n}, flm[-n] (order -m).
// A walk is stable while the values grow or oscillate: it starts at n = l (closed form) and
// ends at the centre n = m cos b of its oscillating range; the walk of order -m covers the
// rest by the same symmetry. Half of the CTA's warps walk orders m >= 0, half the orders -m.
// beta is folded to (0, pi/2] first (d(pi - b)_{m,n} = (-1)^{l+m} d(b)_{m,-n}), where m - n
// and n (1 - cos b) keep t accurate.
// Values below 2^dead (far in the classically forbidden range) are carried as x 2^e and only
// stepped; their products are left out. The exponents are renewed every G steps (G = 4 for
// sin(b/2) >= 2^-16, else 1), between which a value grows by less than 2^(G bits),
// 2^bits > 2 sqrt(2L) cot(b/2); dead = -1021 + G bits is as low as the renewal's factors and the
// value before the last one stay normal numbers. So entries down to 2^(dead + (G-1) bits) keep
// their digits (L = 1024: 2^-972 for b = pi/2, 2^-951 for 0.2, 2^-916 for 0.01): a single
// coefficient gives its column of d. (Summing from 2^-192 on only, beta = 0.2 / 0.8: L = 256
// 43 / 38 us against 39 / 33, whose warps reach the plain loop earlier; L = 1024 620 / 589
// against 619 / 603; L = 2048 4157 / 4042 against 4248 / 4165.)
// A non-finite coefficient makes its degree NaN, as a product with a zero would.
// Grid: (order tiles, degrees from the largest, maps). Six FP64 operations per value and 48 bytes
// of shared-memory broadcasts per step for the R orders of a lane, with no reduction across lanes:
// L = 1024, one float64 map, 0.48-0.62 ms over beta (2.6-3.3 ms with recurrences along the degree,
// whose sums over n crossed lanes, warps and a cluster). ncu there at beta = 1.9: FP64 pipe 53 %,
// shared-memory pipe 52 %, issue 45 %; the barriers between chunks are the first stall, as the
// walks of a CTA end at different steps.
template <typename R2, int R, int G>
__global__ void __launch_bounds__(kWalkThreads, 4) rotate_walk_kernel(RotParams p) {
  // two staged chunks: (A, C) of each step, then its two weights; at the end the exchange
  __shared__ __align__(16) double2 smem[2 * 3 * kWalkThreads];
  double2* const sAC = smem;
  double2* const sX = smem + 2 * kWalkThreads;
  constexpr int kSpan = 32 * R;                          // orders of a warp
  constexpr int kTile = kSpan * (kWalkThreads / 64);     // orders of a CTA
  static_assert(sizeof(smem) >= (size_t)kTile * 4 * sizeof(double), "exchange");
  const int L = p.L, NN = 2 * L - 1, l = L - 1 - (int)blockIdx.y;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const bool neg = warp >= kWalkThreads / 64;            // this warp walks orders -m
  const int mt = blockIdx.x * kTile;
  const int mb = mt + (warp % (kWalkThreads / 64)) * kSpan + lane * R;
  const size_t row = ((size_t)blockIdx.z * L + l) * NN + (L - 1);
  if (mt > l) {  // orders beyond the degree: zeros
    for (int i = tid; i < kTile; i += kWalkThreads)
      if (mt + i < L) {
        RotIO<R2>::put(p.out, row + mt + i, make_double2(0.0, 0.0));
        RotIO<R2>::put(p.out, row - mt - i, make_double2(0.0, 0.0));
      }
    return;
  }
  // start values d_{M,l} = sqrt((2l)! / ((l+M)! (l-M)!)) cos^{l+M} sin^{l-M} of M = +-m
  double v[R], vp[R];
  int e[R];
  int smin = l + 1, smax = -l - 1;  // least and largest last step over the warp
  {
    const RotXD f2 = p.sqf[2 * l];
    const double ig = 1.0 / sqrt(p.w[0] * p.w[2 * l]);
#pragma unroll
    for (int r = 0; r < R; ++r) {
      const int m = mb + r, M = neg ? -m : m;
      v[r] = vp[r] = 0.0;
      e[r] = 0;
      if (m > l) continue;
      const RotXD fa = p.sqf[l + M], fb = p.sqf[l - M], c = p.cpow[l + M], s = p.spow[l - M];
      int d;
      double x = frexp(f2.m / (fa.m * fb.m) * (c.m * s.m) * ig, &d);
      const int ex = f2.e - fa.e - fb.e + c.e + s.e + d;
      if (ex >= p.dead || x == 0.0)
        x = ldexp(x, ex);
      else
        e[r] = ex;
      v[r] = x;
    }
  }
  int last[R];  // last n of each walk
#pragma unroll
  for (int r = 0; r < R; ++r) {
    const int c = (int)ceil((double)(mb + r) * p.cb);
    last[r] = neg ? 1 - c : c;
    if (mb + r <= l) {
      smin = min(smin, last[r]);
      smax = max(smax, last[r]);
    }
  }
  smin = __reduce_min_sync(0xffffffffu, smin);
  smax = __reduce_max_sync(0xffffffffu, smax);
  // the CTA's least last step: that of its largest order's negative walk
  const int mtop = min(l, mt + kTile - 1);
  const int cmin = min((int)ceil((double)mt * p.cb), 1 - (int)ceil((double)mtop * p.cb));
  const int nchunks = (l - cmin) / kWalkThreads + 1;

  double q = (double)((neg ? -mb : mb) - l);  // M - n of the lane's first walk
  double ap[R][2], an[R][2];  // products with flm[n] (order M) and flm[-n] (order -M)
#pragma unroll
  for (int r = 0; r < R; ++r) ap[r][0] = ap[r][1] = an[r][0] = an[r][1] = 0.0;

  // staging: thread tid holds step tid of a chunk
  double2 xr, xl, ph;
  double wa, wb;
  auto fetch = [&](int ch) {
    const int n = l - (ch * kWalkThreads + tid);
    xr = xl = ph = make_double2(0.0, 0.0);
    wa = wb = 0.0;
    if (n >= -l) {
      const int k = p.flip ? -n : n;  // the coefficient that stands for n
      xr = RotIO<R2>::get(p.flm, row + k);
      xl = RotIO<R2>::get(p.flm, row - k);
      ph = p.eg[L - 1 + k];
      wa = p.w[l - n];
      wb = p.w[l + n];
    }
  };
  bool bad = false;
  auto stage = [&](int ch) {
    const int n = l - (ch * kWalkThreads + tid), b = ch & 1;
    const double ww = wa * wb, g = sqrt(ww), dn = (double)n;
    const double A = fma(p.pis, ww, p.pisl * ww);
    const double sp = (p.par & n & 1) ? -g : g;         // (-1)^n where sin, cos differ in sign
    const double sn = ((p.par ^ 1) & n & 1) ? -g : g;   // times the (-1)^n of order -m
    sAC[b * kWalkThreads + tid] = make_double2(A, A * fma(dn, p.y, dn * p.yl));
    double2* const x = sX + 2 * (b * kWalkThreads + tid);
    x[0] = make_double2(sp * (xr.x * ph.x - xr.y * ph.y),
                                 sp * (xr.x * ph.y + xr.y * ph.x));
    x[1] = make_double2(sn * (xl.x * ph.x + xl.y * ph.y),
                                 sn * (xl.y * ph.x - xl.x * ph.y));
    const double z = 0.0 * xr.x + 0.0 * xr.y + 0.0 * xl.x + 0.0 * xl.y;
    bad |= z != z;
  };
  fetch(0);
  stage(0);
  int mode = 0;  // 0: nothing of the warp contributes yet, 1: some lanes do, 2: all do
  if (__any_sync(0xffffffffu, mb <= l && e[0] == 0)) mode = 1;
#pragma unroll
  for (int r = 1; r < R; ++r)
    if (__any_sync(0xffffffffu, mb + r <= l && e[r] == 0)) mode = 1;

  auto renew = [&] {
#pragma unroll
    for (int r = 0; r < R; ++r) {
      if (e[r] < 0) {
        const int x = ((__double2hiint(v[r]) >> 20) & 0x7ff) - 1022, en = e[r] + x;
        const int sh = en >= p.dead ? e[r] : -x;
        const double f = __hiloint2double((1023 + sh) << 20, 0);
        v[r] *= f;
        vp[r] *= f;
        e[r] = en >= p.dead ? 0 : en;
      }
    }
  };
  for (int ch = 0; ch < nchunks; ++ch) {
    __syncthreads();
    const bool more = ch + 1 < nchunks;
    if (more) fetch(ch + 1);
    const int nt = l - ch * kWalkThreads;  // n of the chunk's first step
    const double2* const ac = sAC + (ch & 1) * kWalkThreads;
    const double2* const xx = sX + (ch & 1) * 2 * kWalkThreads;
#pragma unroll 1
    for (int k = 0; k < kWalkThreads && nt - k >= smin; k += G) {
      // one value step of every walk
      auto step = [&](int j) {
        const double2 c = ac[k + j];
        const double t0 = fma(q, c.x, c.y);
        q += 1.0;
#pragma unroll
        for (int r = 0; r < R; ++r) {
          const double t = r == 0 ? t0 : fma(neg ? -(double)r : (double)r, c.x, t0);
          const double x = fma(-t, v[r], -vp[r]);
          vp[r] = v[r];
          v[r] = x;
        }
      };
      if (mode == 2 && nt - k - (G - 1) >= smax) {
#pragma unroll
        for (int j = 0; j < G; ++j) {
          const double2 xp = xx[2 * (k + j)], xn = xx[2 * (k + j) + 1];
#pragma unroll
          for (int r = 0; r < R; ++r) {
            ap[r][0] = fma(v[r], xp.x, ap[r][0]);
            ap[r][1] = fma(v[r], xp.y, ap[r][1]);
            an[r][0] = fma(v[r], xn.x, an[r][0]);
            an[r][1] = fma(v[r], xn.y, an[r][1]);
          }
          step(j);
        }
      } else if (mode == 0) {
#pragma unroll
        for (int j = 0; j < G; ++j) step(j);
        renew();
        bool live = false;
#pragma unroll
        for (int r = 0; r < R; ++r) live |= e[r] == 0 && mb + r <= l;
        if (__any_sync(0xffffffffu, live)) mode = 1;
      } else {
#pragma unroll
        for (int j = 0; j < G; ++j) {
          const double2 xp = xx[2 * (k + j)], xn = xx[2 * (k + j) + 1];
#pragma unroll
          for (int r = 0; r < R; ++r) {
            const double dv = e[r] == 0 && nt - k - j >= last[r] ? v[r] : 0.0;
            ap[r][0] = fma(dv, xp.x, ap[r][0]);
            ap[r][1] = fma(dv, xp.y, ap[r][1]);
            an[r][0] = fma(dv, xn.x, an[r][0]);
            an[r][1] = fma(dv, xn.y, an[r][1]);
          }
          step(j);
        }
        renew();
        bool all = true;
#pragma unroll
        for (int r = 0; r < R; ++r) all &= e[r] == 0;
        if (__all_sync(0xffffffffu, all)) mode = 2;
      }
    }
    if (more) stage(ch + 1);
  }
  bad = __syncthreads_or(bad) || p.nan;

  // the walks of -m hand their sums to those of m, which put both orders together
  double* const ex = reinterpret_cast<double*>(smem);
  const int o0 = mb - mt;
  if (neg) {
#pragma unroll
    for (int r = 0; r < R; ++r) {
      ex[o0 + r] = ap[r][0];
      ex[kTile + o0 + r] = ap[r][1];
      ex[2 * kTile + o0 + r] = an[r][0];
      ex[3 * kTile + o0 + r] = an[r][1];
    }
  }
  __syncthreads();
  if (!neg) {
#pragma unroll
    for (int r = 0; r < R; ++r) {
      const double sg = ((mb + r) & 1) ? -1.0 : 1.0;
      double* const x = ex + o0 + r;
      const double br = x[0], bi = x[kTile], cr = x[2 * kTile], ci = x[3 * kTile];
      x[0] = ap[r][0] + sg * cr;
      x[kTile] = ap[r][1] + sg * ci;
      x[2 * kTile] = br + sg * an[r][0];
      x[3 * kTile] = bi + sg * an[r][1];
    }
  }
  __syncthreads();
  for (int i = tid; i < kTile && mt + i < L; i += kWalkThreads) {
    const int m = mt + i;
    const int odd = (p.par & m) ^ (p.flip & (l + m));
    const double sg = bad ? CUDART_NAN : (odd & 1) ? -1.0 : 1.0;
    const double2 a = p.ea[L - 1 + m];
    double2 u = make_double2(0.0, 0.0), w = u;
    if (m <= l) {
      const double ur = sg * ex[i], ui = sg * ex[kTile + i];
      const double wr = sg * ex[2 * kTile + i], wi = sg * ex[3 * kTile + i];
      u = make_double2(ur * a.x - ui * a.y, ur * a.y + ui * a.x);
      w = make_double2(wr * a.x + wi * a.y, wi * a.x - wr * a.y);
    }
    RotIO<R2>::put(p.out, row + m, u);
    if (m > 0) RotIO<R2>::put(p.out, row - m, w);
  }
}

// rotation with caller-supplied planes dl[l][L-1+m][L-1+n]: one warp per (map, l, m)
template <typename R2>
__global__ void rotate_planes_kernel(RotParams p) {
  const int L = p.L, W = 2 * L - 1, lane = threadIdx.x & 31;
  const long rows = (long)p.batch * L * W;
  const long nwarps = (long)gridDim.x * blockDim.x / 32;
  for (long e = (blockIdx.x * (long)blockDim.x + threadIdx.x) / 32; e < rows; e += nwarps) {
    const int col = (int)(e % W), l = (int)((e / W) % L), b = (int)(e / ((long)W * L));
    const int m = col - (L - 1);
    const size_t row = ((size_t)b * L + l) * W;
    if (m < -l || m > l) {
      if (lane == 0) RotIO<R2>::put(p.out, row + col, make_double2(0.0, 0.0));
      continue;
    }
    const double* P = p.dl_in + ((size_t)l * W + col) * W;  // row m of degree l
    double re = 0.0, im = 0.0;
    for (int n = -l + lane; n <= l; n += 32) {
      const double2 x = RotIO<R2>::get(p.flm, row + L - 1 + n);
      const double2 g = p.eg[L - 1 + n];
      const double d = __ldg(P + L - 1 + n);
      re += d * (x.x * g.x - x.y * g.y);
      im += d * (x.x * g.y + x.y * g.x);
    }
    re = warp_sum(re);
    im = warp_sum(im);
    if (lane == 0) {
      const double2 a = p.ea[L - 1 + m];
      RotIO<R2>::put(p.out, row + col, make_double2(re * a.x - im * a.y, re * a.y + im * a.x));
    }
  }
}

struct RotShape {
  int mt, s, nw, nr;
};

// planes: S n per lane so that at most kRotMaxCluster CTAs of 8 warps cover all 2L-1 n; MT
// (orders per tile) as large as keeps two CTAs per SM busy, with MT x S = 8 recurrences per
// lane at most (16 for L > 4096)
RotShape rotate_shape(int L, int sms) {
  const int NN = 2 * L - 1, slots = (NN + 31) / 32, wmax = kRotThreads / 32;
  RotShape r;
  r.s = 1;
  while ((slots + r.s - 1) / r.s > kRotMaxCluster * wmax) r.s *= 2;
  const int ws = (slots + r.s - 1) / r.s;
  r.nw = ws < wmax ? ws : wmax;
  r.nr = (ws + r.nw - 1) / r.nw;
  if (r.s == 1) {
    r.mt = 8;
    while (r.mt > 2 && (long)r.nr * ((L + r.mt - 1) / r.mt) < 2L * sms) r.mt >>= 1;
    // four orders per tile: twice the CTAs, of 4 warps
    if (r.mt == 4 && r.nw == wmax && 2 * r.nr <= kRotMaxCluster) {
      r.nw /= 2;
      r.nr *= 2;
    }
  } else {
    r.mt = r.s == 2 ? 4 : 2;
  }
  return r;
}

template <int MT, int S>
cudaError_t launch_lrec(const RotParams& p, cudaStream_t s) {
  const size_t nt = 32 * (size_t)p.nw;  // ring and uvq (rotate_lrec_kernel)
  const size_t smem = (size_t)rot_depth<S>() * S * nt * 16 + 2 * kRotChunk * MT * 32;
  void (*kern)(RotParams) = rotate_lrec_kernel<MT, S>;
  const cudaError_t e =
      cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return e;
  kern<<<dim3((unsigned)p.nr, (unsigned)((p.L + MT - 1) / MT)), (unsigned)nt, smem, s>>>(p);
  return cudaGetLastError();
}

cudaError_t planes_launch(RotParams p, cudaStream_t s) {
  const int L = p.L, NN = 2 * L - 1;
  const double c = std::cos(0.5 * p.beta), sn = std::sin(0.5 * p.beta);
  p.cb = std::cos(p.beta);
  p.c2 = c * c;
  p.s2 = sn * sn;
  p.cs2 = (c * sn) * (c * sn);
  p.c_neg = c < 0.0;
  p.s_neg = sn < 0.0;
  int dev = 0, sms = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e == cudaSuccess) e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  if (e != cudaSuccess) return e;
  const RotShape sh = rotate_shape(L, sms);
  p.nw = sh.nw;
  p.nr = sh.nr;
  const long nco = ((long)L * L + 255) / 256;
  rotate_coef_kernel<<<(unsigned)(nco < 8192 ? nco : 8192), 256, 0, s>>>(p);
  const int G = (L + kRotSeg - 1) / kRotSeg, nb = (NN + 127) / 128;
  rotate_start_seg_kernel<<<dim3(nb, G), 128, 0, s>>>(p);
  rotate_start_carry_kernel<<<nb, 128, 0, s>>>(p);
  rotate_start_final_kernel<<<dim3(nb, L), 128, 0, s>>>(p);
  e = cudaGetLastError();
  if (e != cudaSuccess) return e;
  switch (sh.s * 16 + sh.mt) {
    case 16 + 8: return launch_lrec<8, 1>(p, s);
    case 16 + 4: return launch_lrec<4, 1>(p, s);
    case 16 + 2: return launch_lrec<2, 1>(p, s);
    case 32 + 4: return launch_lrec<4, 2>(p, s);
    case 64 + 2: return launch_lrec<2, 4>(p, s);
    case 128 + 2: return launch_lrec<2, 8>(p, s);
    default: return cudaErrorInvalidValue;
  }
}

template <typename R2, int R, int G>
cudaError_t launch_walk(const RotParams& p, cudaStream_t s) {
  constexpr int tile = 16 * R * (kWalkThreads / 32);
  const long grid_z = 65535;  // maps per launch
  for (long b = 0; b < p.batch; b += grid_z) {
    RotParams q = p;
    const size_t off = (size_t)b * p.L * (2 * (size_t)p.L - 1);
    q.flm = static_cast<const R2*>(p.flm) + off;
    q.out = static_cast<R2*>(p.out) + off;
    const unsigned nz = (unsigned)(p.batch - b < grid_z ? p.batch - b : grid_z);
    rotate_walk_kernel<R2, R, G>
        <<<dim3((unsigned)((p.L + tile - 1) / tile), (unsigned)p.L, nz), kWalkThreads, 0, s>>>(q);
  }
  return cudaGetLastError();
}

template <typename R2>
cudaError_t rotate_launch(RotParams p, cudaStream_t s) {
  const int L = p.L, NN = 2 * L - 1;
  // beta folded to b in (0, pi/2]: cos and sin of b/2 in double-double
  long double c = cosl(0.5L * p.beta), sn = sinl(0.5L * p.beta);
  p.nan = !std::isfinite(p.beta);
  if (p.nan) c = sn = 0.70710678118654752440L;
  p.par = (c < 0.0L) != (sn < 0.0L);
  c = fabsl(c);
  sn = fabsl(sn);
  p.flip = c < sn;
  if (p.flip) std::swap(c, sn);
  // below 2^-500 (the factors 2^bits of a step would leave the double range) the rotation is the
  // identity: its values run on 2^-500 and all that is not near 1 is left out
  const bool ident = sn < ldexpl(1.0L, -500);
  if (ident) sn = ldexpl(1.0L, -500);
  p.ch = (double)c;
  p.cl = (double)(c - p.ch);
  p.sh = (double)sn;
  p.sl = (double)(sn - p.sh);
  p.cb = (double)((c - sn) * (c + sn));
  // hi + lo: a rounding of these would be the same in every step and add up along the walk
  const long double y = 2.0L * sn * sn, pis = 3.14159265358979323846264338L / (2.0L * sn * c);
  p.y = (double)y;
  p.yl = (double)(y - p.y);
  p.pis = (double)pis;
  p.pisl = (double)(pis - p.pis);
  const int n = p.dl_in ? NN : 2 * L;
  rotate_tables_kernel<<<(n + kRotTab - 1) / kRotTab + (p.dl_in ? 0 : 1), kRotTab, 0, s>>>(p);
  const cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return e;
  if (p.dl_in) {
    const long warps = (long)p.batch * L * NN;
    long blocks = (warps + 7) / 8;
    if (blocks > 65535L * 16) blocks = 65535L * 16;
    rotate_planes_kernel<R2><<<(unsigned)blocks, 256, 0, s>>>(p);
    return cudaGetLastError();
  }
  const int G = sn < 0x1p-16L ? 1 : 4;
  p.dead = ident ? -400 : -1021 + G * (int)ceill(log2l(2.0L * sqrtl(2.0L * L) * c / sn));
  if (G == 1) return launch_walk<R2, 2, 1>(p, s);
  // two orders per lane leave enough warps up to here (L = 1024, beta = 0.2 / 1.5: 626 / 485 us
  // against 664 / 473 with four; L = 1500: 1784 / 1412 against 1803 / 1340), four need fewer
  // broadcasts per order beyond (L = 2048: 4155 / 3222 us against 4282 / 3463)
  return L < 1600 ? launch_walk<R2, 2, 4>(p, s) : launch_walk<R2, 4, 4>(p, s);
}

}  // namespace

static size_t rot_align(size_t b) { return (b + 255) & ~(size_t)255; }

size_t rotate_workspace_bytes(int L) {
  RotParams p{};
  p.L = L;
  return rotate_bind_workspace(p, nullptr);
}

size_t rotate_bind_workspace(RotParams& p, void* ws) {
  const size_t L = (size_t)p.L, NN = 2 * L - 1, G = (L + kRotSeg - 1) / kRotSeg;
  char* const base = static_cast<char*>(ws);
  size_t off = 0;
  auto carve = [&](auto*& x, size_t n) {
    x = reinterpret_cast<std::remove_reference_t<decltype(x)>>(base + off);
    off += rot_align(n * sizeof(*x));
  };
  carve(p.ea, NN);
  carve(p.eg, NN);
  carve(p.w, 2 * L);
  carve(p.sqf, 2 * L);
  carve(p.cpow, 2 * L);
  carve(p.spow, 2 * L);
  carve(p.T, L * L);
  carve(p.UVQ, L * L);
  carve(p.start, L * NN);
  carve(p.carry, G * NN);
  return off;
}

cudaError_t launch_rotate(bool fp64, const RotParams& p, cudaStream_t s) {
  if (!p.flm) return planes_launch(p, s);
  return fp64 ? rotate_launch<double2>(p, s) : rotate_launch<float2>(p, s);
}

}  // namespace s2b

// ----------------------------------------------------------------------------
// C ABI
// ----------------------------------------------------------------------------
extern "C" {

size_t s2b_rotate_workspace_size(int L) { return L >= 1 ? s2b::rotate_workspace_bytes(L) : 0; }

int s2b_rotate_flms(int L, int batch, int precision, double alpha, double beta, double gamma,
                    const void* flm, void* out, const double* dl, void* ws, size_t ws_bytes,
                    void* stream) {
  if (L < 1 || batch < 1 || !flm || !out || !ws)
    return s2b::set_last_error(S2B_ERR_INVALID, "rotate: L >= 1, batch >= 1 and non-NULL buffers");
  if (!dl && L > s2b::kRotMaxL)
    return s2b::set_last_error(S2B_ERR_INVALID, "rotate: L <= 8192 unless the planes are given");
  if (flm == out)
    return s2b::set_last_error(S2B_ERR_INVALID, "rotate: out must not alias flm");
  if (precision != S2B_F64 && precision != S2B_F32)
    return s2b::set_last_error(S2B_ERR_INVALID, "rotate: precision must be S2B_F64 or S2B_F32");
  if (ws_bytes < s2b::rotate_workspace_bytes(L))
    return s2b::set_last_error(S2B_ERR_WORKSPACE, "rotate: workspace too small");
  s2b::RotParams p{};
  p.L = L;
  p.batch = batch;
  p.alpha = alpha;
  p.beta = beta;
  p.gamma = gamma;
  p.flm = flm;
  p.out = out;
  p.dl_in = dl;
  s2b::rotate_bind_workspace(p, ws);
  const cudaError_t e =
      s2b::launch_rotate(precision == S2B_F64, p, reinterpret_cast<cudaStream_t>(stream));
  if (e != cudaSuccess) return s2b::set_last_error(S2B_ERR_CUDA, cudaGetErrorString(e));
  return S2B_OK;
}

int s2b_rotate_dls(int L, double beta, double* dl, void* ws, size_t ws_bytes, void* stream) {
  if (L < 1 || !dl || !ws)
    return s2b::set_last_error(S2B_ERR_INVALID, "rotate_dls: L >= 1 and non-NULL buffers");
  if (L > s2b::kRotMaxL)
    return s2b::set_last_error(S2B_ERR_INVALID, "rotate_dls: L <= 8192");
  if (ws_bytes < s2b::rotate_workspace_bytes(L))
    return s2b::set_last_error(S2B_ERR_WORKSPACE, "rotate_dls: workspace too small");
  s2b::RotParams p{};
  p.L = L;
  p.batch = 0;
  p.beta = beta;
  p.dl_out = dl;
  s2b::rotate_bind_workspace(p, ws);
  const cudaError_t e = s2b::launch_rotate(true, p, reinterpret_cast<cudaStream_t>(stream));
  if (e != cudaSuccess) return s2b::set_last_error(S2B_ERR_CUDA, cudaGetErrorString(e));
  return S2B_OK;
}

}  // extern "C"
