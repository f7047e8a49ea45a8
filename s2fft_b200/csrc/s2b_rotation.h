// Rotation of spherical-harmonic coefficients (rotation.cu).
#pragma once

#include <cuda_runtime.h>

#include <cstddef>

namespace s2b {

constexpr int kRotThreads = 256;     // threads per CTA at most (8 warps)
constexpr int kRotMaxCluster = 8;    // CTAs of an order tile (planes)
constexpr int kRotMaxL = 8192;       // largest band-limit of the recurrence path

// a double with a separate binary exponent: m * 2^e (m in [0.5, 1) or 0), or a start
// value v * 2^k of the recurrence (k < 0 only below 2^-960)
struct RotXD {
  double m;
  int e;
  int pad;
};

struct RotParams {
  int L, batch;
  double alpha, beta, gamma;
  const void* flm;      // [batch][L][2L-1] coefficients (nullptr: planes only)
  void* out;            // [batch][L][2L-1] rotated coefficients
  const double* dl_in;  // caller planes [L][2L-1][2L-1] at beta (nullptr: recurrence)
  double* dl_out;       // planes written in that layout (every entry, zeros included)
  // planes: cos(beta), c^2, s^2, (cs)^2 with c = cos(beta/2), s = sin(beta/2), and the signs
  // of c, s; rotation: cos(b) of the folded angle b in (0, pi/2]
  double cb, c2, s2, cs2;
  int c_neg, s_neg;
  // rotation: cos(b/2), sin(b/2), 1 - cos(b), pi / sin(b) as hi + lo
  double ch, cl, sh, sl, y, yl, pis, pisl;
  int flip;             // beta stands for pi - b
  int par;              // d of beta has the further sign (-1)^{m-n}
  int nan;              // beta is not finite
  int dead;             // the walk's values below 2^dead are not summed
  // workspace (rotate_bind_workspace):
  double2* ea;     // exp(-i m alpha), m in [-(L-1), L-1]
  double2* eg;     // exp(-i n gamma)
  double* w;       // [2L] W(j) of the walk along n
  RotXD* sqf;      // [2L] sqrt(k!)
  RotXD* cpow;     // [2L] cos(b/2)^k
  RotXD* spow;     // [2L] sin(b/2)^k
  double2* T;      // [L][L] (1/sqrt((l+1)^2-k^2), sqrt(l^2-k^2)) for k <= l, else 0
  double4* UVQ;    // [L][L] ((l+1)(2l+1) T.x, T.y/(l(2l+1)), -m/(l(l+1)), 0) for m <= l, else 0
  RotXD* start;    // [L][2L-1] d^{l}_{l,a}(beta) at [l][L-1+a], |a| <= l
  RotXD* carry;    // [ceil(L/32)][2L-1] segment products of the start table
  // launch shape of the planes kernel: warps per CTA and CTAs per order tile
  int nw, nr;
};

size_t rotate_workspace_bytes(int L);
// carves the workspace into the tables; returns its size
size_t rotate_bind_workspace(RotParams& p, void* ws);
cudaError_t launch_rotate(bool fp64, const RotParams& p, cudaStream_t s);

}  // namespace s2b
