// Complex transforms of lines whose length is not a power of two (FFTW plans any
// length, compute_potential.c:247-309), FP64: mixed-radix Stockham passes between
// two shared-memory copies of a block's lines. Radices 8, 4, 2, 3, 5, 7, 11 and 13
// are butterflies in registers, a larger prime p is summed directly, one output
// per thread (p terms). Twiddles exp(-2 pi i m / N) come from the host's table.
//
// The sums over whole lines that these replace take N terms a point; a pass takes
// its radix. Bound: shared memory, one read and one write of 16 bytes a point and
// pass. Measured at 96 x 180 x 120 per launch, direct -> mixed: divergence and y
// transform 0.29 -> 0.053 ms, z 0.17 -> 0.023, inverse y 0.27 -> 0.035.
#pragma once
#include "tc_common.cuh"

namespace tcgpu {

// the passes of a length, in order
struct Radices {
  int count;
  unsigned short r[12];
};
inline Radices radices_of(int n) {
  Radices p{};
  auto take = [&](int f) {
    while (n % f == 0 && n > 1) {
      p.r[p.count++] = (unsigned short)f;
      n /= f;
    }
  };
  for (int f : {8, 4, 2, 3, 5, 7, 11, 13}) take(f);
  for (int f = 17; f * f <= n; f += 2) take(f);
  if (n > 1) p.r[p.count++] = (unsigned short)n;
  return p;
}

__device__ __forceinline__ double2 mix_mul(double2 a, double2 b) {
  return make_double2(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x);
}
template <int SIGN>
__device__ __forceinline__ double2 mix_tw(const double2 * __restrict__ tw, int m) {
  double2 w = __ldg(tw + m);
  if (SIGN > 0) w.y = -w.y;
  return w;
}

// v[s] <- sum_r v[r] exp(SIGN 2 pi i r s / R) for odd R: cosines and sines of
// 2 pi k / R from the table (entry k N / R), pairs r and R - r combined
template <int R, int SIGN>
__device__ __forceinline__ void dft_odd(double2 (&v)[R], const double2 * __restrict__ tw, int NR) {
  constexpr int H = (R - 1) / 2;
  double2 t[H + 1], u[H + 1], c[H + 1];
#pragma unroll
  for (int k = 1; k <= H; k++) {
    t[k] = make_double2(v[k].x + v[R - k].x, v[k].y + v[R - k].y);
    u[k] = make_double2(v[k].x - v[R - k].x, v[k].y - v[R - k].y);
    c[k] = __ldg(tw + k * NR);
    c[k].y = SIGN < 0 ? -c[k].y : c[k].y;   // sin(2 pi k / R) for SIGN < 0, minus it for SIGN > 0
  }
  const double2 v0 = v[0];
  double2 s0 = v0;
#pragma unroll
  for (int k = 1; k <= H; k++) { s0.x += t[k].x; s0.y += t[k].y; }
  v[0] = s0;
#pragma unroll
  for (int s = 1; s <= H; s++) {
    double ax = v0.x, ay = v0.y, bx = 0., by = 0.;
#pragma unroll
    for (int k = 1; k <= H; k++) {
      const int q = (k * s) % R, f = q <= H ? q : R - q;
      const double sn = q <= H ? c[f].y : -c[f].y;
      ax += t[k].x * c[f].x;
      ay += t[k].y * c[f].x;
      bx += u[k].x * sn;
      by += u[k].y * sn;
    }
    // X_s = A - i B, X_{R-s} = A + i B
    v[s] = make_double2(ax + by, ay - bx);
    v[R - s] = make_double2(ax - by, ay + bx);
  }
}
template <int R, int SIGN>
__device__ __forceinline__ void dft_small(double2 (&v)[R], const double2 * __restrict__ tw, int NR) {
  if constexpr (R == 2) {
    const double2 a = v[0], b = v[1];
    v[0] = make_double2(a.x + b.x, a.y + b.y);
    v[1] = make_double2(a.x - b.x, a.y - b.y);
  } else if constexpr (R == 4) {
    const double2 a = make_double2(v[0].x + v[2].x, v[0].y + v[2].y), b = make_double2(v[0].x - v[2].x, v[0].y - v[2].y);
    const double2 c = make_double2(v[1].x + v[3].x, v[1].y + v[3].y), d = make_double2(v[1].x - v[3].x, v[1].y - v[3].y);
    const double2 e = SIGN < 0 ? make_double2(d.y, -d.x) : make_double2(-d.y, d.x);   // SIGN i d
    v[0] = make_double2(a.x + c.x, a.y + c.y);
    v[1] = make_double2(b.x + e.x, b.y + e.y);
    v[2] = make_double2(a.x - c.x, a.y - c.y);
    v[3] = make_double2(b.x - e.x, b.y - e.y);
  } else if constexpr (R == 8) {
    double2 o[4] = {v[1], v[3], v[5], v[7]}, e[4] = {v[0], v[2], v[4], v[6]};
    dft_small<4, SIGN>(e, tw, NR);
    dft_small<4, SIGN>(o, tw, NR);
    constexpr double h = 0.70710678118654752;
    const double2 w1 = make_double2(h, SIGN * h), w2 = make_double2(0., (double)SIGN), w3 = make_double2(-h, SIGN * h);
    o[1] = mix_mul(o[1], w1);
    o[2] = mix_mul(o[2], w2);
    o[3] = mix_mul(o[3], w3);
#pragma unroll
    for (int s = 0; s < 4; s++) {
      v[s] = make_double2(e[s].x + o[s].x, e[s].y + o[s].y);
      v[s + 4] = make_double2(e[s].x - o[s].x, e[s].y - o[s].y);
    }
  } else {
    dft_odd<R, SIGN>(v, tw, NR);
  }
}

// element e of a padded line (as the power-of-two transforms pad theirs)
__device__ __forceinline__ int mpad(int i) { return i + (i >> 4); }
// slots of a padded line, odd, so that neighbouring lines start on other banks
__host__ __device__ constexpr int mixed_len(int n) { return (n + (n >> 4)) | 1; }

// Every butterfly of one pass of radix R over P lines: inputs x[p, j + r N / R]
// through ld(p, e), outputs through st(p, e, v). PFAST: lanes run along the lines
// (P a power of two), otherwise along the elements.
template <int R, int SIGN, bool PFAST, class Ld, class St>
__device__ __forceinline__ void mixed_pass(int N, int Ns, int P, const double2 * __restrict__ tw, const Ld & ld,
                                           const St & st) {
  const int NR = N / R, ts = NR / Ns;
  for (int u = threadIdx.x; u < P * NR; u += blockDim.x) {
    const int p = PFAST ? u & (P - 1) : u / NR, j = PFAST ? u / P : u - p * NR;
    const int k = j % Ns, base = (j - k) * R + k;
    double2 v[R];
#pragma unroll
    for (int r = 0; r < R; r++) v[r] = ld(p, j + r * NR);
    if (Ns > 1) {
#pragma unroll
      for (int r = 1; r < R; r++) v[r] = mix_mul(v[r], mix_tw<SIGN>(tw, r * k * ts));
    }
    dft_small<R, SIGN>(v, tw, NR);
#pragma unroll
    for (int r = 0; r < R; r++) st(p, base + r * Ns, v[r]);
  }
}
// the same for a prime R without a butterfly: one output per thread
template <int SIGN, bool PFAST, class Ld, class St>
__device__ __forceinline__ void prime_pass(int R, int N, int Ns, int P, const double2 * __restrict__ tw, const Ld & ld,
                                           const St & st) {
  const int NR = N / R, ts = NR / Ns;
  for (int u = threadIdx.x; u < P * N; u += blockDim.x) {
    const int p = PFAST ? u & (P - 1) : u / N, o = PFAST ? u / P : u - p * N;
    const int s = o / NR, j = o - s * NR, k = j % Ns;
    const int inc = (k * ts + s * NR) % N;   // twiddle of x[j + r N / R]: r inc
    double2 a = make_double2(0., 0.);
    int q = 0;
    for (int r = 0; r < R; r++) {
      const double2 x = ld(p, j + r * NR), w = mix_tw<SIGN>(tw, q);
      a.x += x.x * w.x - x.y * w.y;
      a.y += x.x * w.y + x.y * w.x;
      q += inc;
      if (q >= N) q -= N;
    }
    st(p, (j - k) * R + k + s * Ns, a);
  }
}

// Transforms of P lines of N points: the first pass reads through ld, the last one
// writes through st, the others go between the shared copies a and b (lines LS
// slots apart). The caller synchronises before ld's data are needed and after st's.
template <int SIGN, bool PFAST, class Ld, class St>
__device__ void mixed_fft(const Radices & rd, int N, int P, double2 * a, double2 * b, int LS,
                          const double2 * __restrict__ tw, const Ld & ld, const St & st) {
  int Ns = 1;
  for (int q = 0; q < rd.count; q++) {
    const int R = rd.r[q];
    const bool first = q == 0, last = q == rd.count - 1;
    double2 * from = (q & 1) ? a : b, * to = (q & 1) ? b : a;
    auto in = [&](int p, int e) { return first ? ld(p, e) : from[p * LS + mpad(e)]; };
    auto out = [&](int p, int e, double2 v) {
      if (last) st(p, e, v);
      else to[p * LS + mpad(e)] = v;
    };
    switch (R) {
      case 2: mixed_pass<2, SIGN, PFAST>(N, Ns, P, tw, in, out); break;
      case 3: mixed_pass<3, SIGN, PFAST>(N, Ns, P, tw, in, out); break;
      case 4: mixed_pass<4, SIGN, PFAST>(N, Ns, P, tw, in, out); break;
      case 5: mixed_pass<5, SIGN, PFAST>(N, Ns, P, tw, in, out); break;
      case 7: mixed_pass<7, SIGN, PFAST>(N, Ns, P, tw, in, out); break;
      case 8: mixed_pass<8, SIGN, PFAST>(N, Ns, P, tw, in, out); break;
      case 11: mixed_pass<11, SIGN, PFAST>(N, Ns, P, tw, in, out); break;
      case 13: mixed_pass<13, SIGN, PFAST>(N, Ns, P, tw, in, out); break;
      default: prime_pass<SIGN, PFAST>(R, N, Ns, P, tw, in, out); break;
    }
    Ns *= R;
    if (!last) __syncthreads();
  }
}

}  // namespace tcgpu
