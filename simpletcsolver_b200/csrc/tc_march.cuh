// The marching predict kernel (fluid_predict_field, src/fluid/predict/main.c:35-110)
// as templates; tc_march*.cu instantiate it, tc_march.cu chooses the instance.
//
// One pass over the fields per substep: right-hand sides of ux (face i), uy,
// uz, t (centre i), the new explicit source terms, the RK increment
// delta = dt (alpha srcA + beta srcA_prev + gamma srcG) with srcG (implicit
// diffusion + pressure gradient) kept in registers, the radial implicit solve
// (src/tdm.c:17-50), and u + delta into the other buffer of the pair with walls
// and periodic images (boundary/*.c, halo.c).
//
// A CTA owns JT neighbouring radial lines (j0 .. j0 + JT - 1, PAIRS pairs) and
// marches through KC planes in z. A ring of four plane slots in shared memory
// holds the rows j0-1 .. j0+JT of ux, uy, uz, t and j0-1 .. j0+JT-1 of p; the
// previous substep's source terms of the CTA's lines arrive in a two-plane
// buffer of their own. Roles, which meet only at mbarriers:
//   field warps (NFW)  group A: ux at face i and t at centre i of a line pair,
//                      group B: uy and uz at centre i; a warp has one group
//                      (NG = 2) or both (NG = 1)
//   solve warps (4)    variable v of every line: radial solve, update, stores of
//                      the new fields (or of the increments), and its copies
//                      into the ring and the old terms
// The field warps hand a plane's increments to the solve warps through a
// double-buffered staging area and never wait for the solutions.
//
// What bounds it: the solve warps' serial chain, with the field warps close
// behind. The kernel moves 104 / 136 bytes a cell (the first / later substeps),
// 2.2 / 2.8 ms at 256 x 1024 x 512 at the copy bandwidth, and its FP64 instructions
// need about 1.2 ms of the FP64 pipe; at nx = 256 a plane of two lines takes a
// solve warp about 4.0 thousand cycles (clock64 around each part, 256 x 512 x 128):
// 1.55 the two solves (dependent FP64 and shuffle latencies), 0.78 issuing copies,
// 1.16 the update and the stores, 0.45 waits. One CTA of 12 warps fits an SM: 8 field warps with both groups at
// 176 registers and 4 solve warps at 152, none spilling. 16 field warps at 96
// registers spill and are slower (1.80 against 1.09 ms at 256 x 512 x 256), as are
// solves whose scans run half as far (30.7 against 27.1 ps a cell). Per launch
// 6.8 -> 3.8 ms at 256 x 1024 x 512 against the form whose field warps solved,
// updated and stored.
//
// Every face between two cells of a thread is formed once: the thread carries
// the z face's share of the next plane's cell in registers (so plane k - 1 is
// read only where a term spans both planes), and the y face between the two
// lines of a pair serves both.
//
// The rows j0-1 .. j0+JT of a field are consecutive in memory, and an even
// number of rows (j0 is odd, ny even) starts them on a 16-byte boundary, so one
// bulk copy per field and plane moves them all (issuing a copy costs its warp
// about 90 cycles: one copy per row, 23 a plane, took a third of the march).
// Rows in shared memory are then as far apart as in memory. Tiles, parts of rows
// longer than 256 points, take one copy per row, widened to 16-byte bounds.
#pragma once
#include <type_traits>

#include "tc_common.cuh"
#include "tc_kernels.h"

namespace tcgpu {
namespace march {

#define LD(p) __ldg(p)
__device__ __forceinline__ void prefetch_l1(const void * p) { asm volatile("prefetch.global.L1 [%0];" ::"l"(p)); }

// Shared memory, in bytes, shared by the kernel and its launcher. Row buffers
// are sized for the widest radial line of the warp count (nx <= 32 NW), so
// every stencil offset is a compile-time constant.
template <int NW_, int PAIRS_, int NG_, class T>
struct Layout {
  static constexpr int NW = NW_, PAIRS = PAIRS_, NG = NG_;
  static constexpr bool D64 = sizeof(T) == 8;
  static constexpr int E = NW;                      // elements per lane of the radial solves
  static constexpr int JT = 2 * PAIRS;              // lines per CTA
  static constexpr int NT = 32 * NW;                // radial indices per CTA
  static constexpr int NFW = NG * NW * PAIRS;       // field warps: a warp per group, or one for both (NG = 1)
  static constexpr int NSW = 4;                     // solve warps
  static constexpr int THREADS = 32 * (NFW + NSW);
  // The roles split the registers of the launch (setmaxnreg; the warpgroups'
  // shares add up to the launch total), so that none of them spills: the rest of
  // the L1 is too small to hold spilled values, which then come from the L2 (8
  // warps of 200 registers and 4 of 104, whose solves spill: 1.80 ms at
  // 256 x 512 x 256; 176 and 152: 1.09 ms).
  static constexpr bool SPLIT8 = NFW == 8, SPLIT12 = NFW == 12 && E > 4;
  static constexpr int REGS = SPLIT8 ? 168 : SPLIT12 ? 128 : 0;
  static constexpr int REGS_FIELD = SPLIT8 ? 176 : SPLIT12 ? 120 : 0, REGS_SOLVE = SPLIT8 || SPLIT12 ? 152 : 0;
  static_assert(NFW * REGS_FIELD + NSW * REGS_SOLVE <= (NFW + NSW) * REGS, "register split");
  static constexpr int NR = JT + 2;                 // rows per field
  // A slot's blocks (elements of T): ux, uy, uz, t, then p in double. Rows are
  // S elements apart, S = nx + 2 (double) or the padded pitch (float), ux rows of
  // nx + 1 doubles S - 1; sized here for the widest line of the warp count. Tiles
  // use S = RL (RL + 1 in double and in p for odd nx) and ux rows S + 1 apart, so
  // that consecutive rows keep the parity of their starts in memory.
  static constexpr int RL = 32 * NW + 4;
  static constexpr int FBS = NR * (RL + 2);         // a block
  __host__ __device__ static constexpr int FB(int f) { return f * FBS; }
  static constexpr size_t POFF = (size_t)4 * FBS * sizeof(T);
  static constexpr size_t SLOT = (POFF + (size_t)((JT + 1) * (RL + 1) + 2) * sizeof(double) + 15) & ~(size_t)15;
  static_assert(FBS % 2 == 0 && POFF % 16 == 0, "blocks start on 16-byte boundaries");
  static constexpr int NSLOT = 4;                   // planes k - 1 .. k + 2
  static constexpr int SL = 32 * E + 32;            // staging line (padded for the solves)
  static constexpr size_t STAGE = NSLOT * SLOT;     // [2][JT][4][SL] doubles after the ring
  static constexpr int OL = 32 * NW;                // old source terms per line and variable
  static constexpr size_t OLDS = STAGE + sizeof(double) * 2 * JT * 4 * SL;   // [2][4][JT OL] T
  static constexpr size_t BAR = OLDS + sizeof(T) * 2 * 4 * JT * OL;
  // mbarriers: ring slots full / empty, staging full[2] / empty[2], old terms[2]
  static constexpr int NBAR = 2 * NSLOT + 6;
  static constexpr size_t BYTES = BAR + NBAR * sizeof(unsigned long long) + 16;   // + the abort flag
  static_assert(STAGE % 16 == 0 && OLDS % 16 == 0 && BAR % 8 == 0, "alignment");
  static_assert(BYTES <= 232448, "shared memory");
};

// Everything the roles need besides their coefficients.
template <class T>
struct Args {
  Geo g;
  Bc bc;
  Coefs cf;
  XFactors xf;
  double nu, kappa;
  FieldsT<T> in, out;
  SrcSetT<T> ss;
  DeltaSet ds;
  int rkstep, mode, KC;
  unsigned * status;
  unsigned lost;   // bytes announced with every plane that no copy brings: 0 but in the self-test of the waits
};

__device__ __forceinline__ void mbar_arrive(unsigned long long * bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}
// Bounded wait of one thread; after any wait of the CTA has given up, nobody waits any
// more: the CTA runs to its end, arriving as ever, without copying or storing fields any
// more (source terms it still stores; they belong to a step that is reported as failed,
// and a look at the flag before each store costs up to 3.5% of the kernel). The lanes of a
// warp may find out at different times, so a branch on the flag holds no operation of a
// whole warp (__syncwarp, shuffles) unless the warp has voted on it.
__device__ __forceinline__ bool await(unsigned long long * bar, unsigned parity, volatile int * abort_flag) {
  if (mbar_try_wait(bar, parity)) return true;
  const long long t0 = clock64();
  while (!mbar_try_wait(bar, parity)) {
    if (*abort_flag) return false;
    if (clock64() - t0 > kWaitCycles) {
      *abort_flag = 1;
      return false;
    }
  }
  return true;
}

// The barriers of a CTA.
template <class L>
struct Bars {
  unsigned long long * b;
  __device__ unsigned long long * full(int slot) const { return b + slot; }
  __device__ unsigned long long * empty(int slot) const { return b + L::NSLOT + slot; }
  __device__ unsigned long long * staged(int q) const { return b + 2 * L::NSLOT + q; }
  __device__ unsigned long long * unstaged(int q) const { return b + 2 * L::NSLOT + 2 + q; }
  __device__ unsigned long long * olds(int q) const { return b + 2 * L::NSLOT + 4 + q; }
};

// ------------------------------------------------------------ coefficients
// Products of the metric tables taken once on the host (the P_* tables), each
// spelled out below where it is used; loaded once per thread (they depend on i
// only) with the diffusivities folded in. (FP32-storage contexts have sides of
// their own: tc_march_f32.cuh.)
template <class C>
struct CoefA {
  C xa1, xa2, xa3, yb1, yb2, zc1, zc2, h1, h2;        // ux advection, centrifugal term
  C lxl, lxu, ly;                                     // ux Laplacian, x (carry 2 nu) and y (nu)
  C cy1, cy2, ca1, ca2, cz1, px;                      // ux cross diffusion (carry nu), pressure gradient
  C tx0, tx1, ty, kl, ku, ky;                         // t advection, Laplacian in x and y (carry kappa)
};
template <class C>
struct CoefB {
  C a1, a2, b, h;                                     // uy / uz advection
  C lxl, lxu, ly;                                     // centred Laplacian, x and y (carry nu)
  C p1, p2, qm, q0, qp, yk, yz, py;                   // uy cross diffusion (carry nu), pressure gradient
  C zx0, zx1;                                         // uz cross diffusion (carry nu; its y term shares yz)
};
// radially uniform coefficients: z Laplacian 1/hz^2 times nu, kappa; 0.5/hz, 0.25/hz, 1/hz
template <class C>
struct CoefZ {
  C nz, kz, t, c, ih;
};
// The Laplacians are applied as differences from the centre value: the centre
// coefficients of the tables are the negated sums of the others (F_LXC =
// -F_LXL - F_LXU, F_LYC = -2 F_LYL = -2 F_LYU, likewise for C_* and in z), so
// l a + c b + u d = l (a - b) + u (d - b) and only l and u are held.
template <class C>
__device__ __forceinline__ void load_coefs(CoefA<C> & q, const Coefs & cf, int i, double nu, double kappa) {
  const double * __restrict__ b = cf.tab + i;
#define CF(T) LD(b + (T) * CSTRIDE)
  q.xa1 = (C)CF(P_XA1); q.xa2 = (C)CF(P_XA2); q.xa3 = (C)CF(P_XA3);
  q.yb1 = (C)CF(P_YB1); q.yb2 = (C)CF(P_YB2); q.zc1 = (C)CF(P_ZC1); q.zc2 = (C)CF(P_ZC2);
  q.h1 = (C)CF(P_H1); q.h2 = (C)CF(P_H2);
  q.lxl = (C)CF(F_LXL) * (C)(2. * nu); q.lxu = (C)CF(F_LXU) * (C)(2. * nu); q.ly = (C)CF(F_LYL) * (C)nu;
  q.cy1 = (C)CF(P_CY1) * (C)nu; q.cy2 = (C)CF(P_CY2) * (C)nu;
  q.ca1 = (C)CF(P_CA1) * (C)nu; q.ca2 = (C)CF(P_CA2) * (C)nu; q.cz1 = (C)CF(P_CZ1) * (C)nu;
  q.px = (C)CF(C_INVHXXF);
  q.tx0 = (C)CF(P_TX0); q.tx1 = (C)CF(P_TX1); q.ty = (C)CF(P_TY);
  q.kl = (C)CF(C_LXL) * (C)kappa; q.ku = (C)CF(C_LXU) * (C)kappa; q.ky = (C)CF(C_LYL) * (C)kappa;
}
template <class C>
__device__ __forceinline__ void load_coefs(CoefB<C> & q, const Coefs & cf, int i, double nu, double) {
  const double * __restrict__ b = cf.tab + i;
  q.a1 = (C)CF(P_UA1); q.a2 = (C)CF(P_UA2); q.b = (C)CF(P_UB); q.h = (C)CF(P_UH);
  q.lxl = (C)CF(C_LXL) * (C)nu; q.lxu = (C)CF(C_LXU) * (C)nu; q.ly = (C)CF(C_LYL) * (C)nu;
  q.p1 = (C)CF(P_P1) * (C)nu; q.p2 = (C)CF(P_P2) * (C)nu;
  q.qm = (C)CF(P_QM) * (C)nu; q.q0 = (C)CF(P_Q0) * (C)nu; q.qp = (C)CF(P_QP) * (C)nu;
  q.yk = (C)CF(P_YK) * (C)nu; q.yz = (C)CF(P_YZ) * (C)nu; q.py = (C)CF(C_INVHYXC);
  q.zx0 = (C)CF(P_ZX0) * (C)nu; q.zx1 = (C)CF(P_ZX1) * (C)nu;
#undef CF
}

// Element of face i, row r (cell offset i - ib), relative to a centre row's
// element: double: face i is element i - 1 of a row of one element less; in a
// tile the rows are one element longer and start two faces early.
template <class T, bool TILE>
__host__ __device__ constexpr int ux_shift(int r) { return sizeof(T) == 4 ? 0 : TILE ? r + 1 : -r - 1; }
// A thread's view of one plane slot: bases already moved to the thread's radial
// index and line pair.
template <class L, class T, bool TILE>
struct View {
  const T * f;        // ux
  const T * c;        // centre fields
  const double * p;
  int s, sp;          // elements between rows of T, of p
};
// row r = 0 .. 3 of the pair: j - 1 + r for the pair's first line j
#define UX(V, r, di) (C)(V).f[(r) * (V).s + L::FB(0) + ux_shift<T, TILE>(r) + (di)]
#define UY(V, r, di) (C)(V).c[(r) * (V).s + L::FB(1) + (di)]
#define UZ(V, r, di) (C)(V).c[(r) * (V).s + L::FB(2) + (di)]
#define TT(V, r, di) (C)(V).c[(r) * (V).s + L::FB(3) + (di)]
#define PP(V, r, di) (V).p[(r) * (V).sp + (di)]

// IMPL: the implicit directions as a compile-time mask (bit 0 x, 1 y, 2 z), plus
// 8 with the closure forcing; or the run-time flags, -1 without and -2 with forcing
__host__ __device__ constexpr bool forced(int impl) { return impl == -2 || (impl >= 0 && (impl & 8) != 0); }
template <int IMPL>
struct Dirs {
  bool x, y, z;
  __device__ explicit Dirs(const Bc & bc)
      : x(IMPL >= 0 ? (IMPL & 1) != 0 : bc.implicit[0] != 0), y(IMPL >= 0 ? (IMPL & 2) != 0 : bc.implicit[1] != 0),
        z(IMPL >= 0 ? (IMPL & 4) != 0 : bc.implicit[2] != 0) {}
};

// Every multiply-add of the right-hand sides is spelled out, so that the rounding
// of a term does not depend on the instance (compile-time or run-time directions,
// with or without forcing) it is compiled in.
__device__ __forceinline__ double mad(double a, double b, double c) { return fma(a, b, c); }
__device__ __forceinline__ float mad(float a, float b, float c) { return fmaf(a, b, c); }

// shares of a z face in the explicit (e) and implicit (g) sides of a variable of both lines
template <class C>
struct Share {
  C e[2], g[2];
};

// The z face between a plane's cell (value lo) and the next one's (hi) of one
// variable: flux F (already 0.5 / volume times the advecting flux), diffusion
// coefficient nz. Skew-symmetric advection and diffusion add
// (F - nz)(lo - hi) to the lower cell and (F + nz)(lo - hi) to the upper one;
// with z implicit the diffusive part goes to the implicit side.
template <class C>
__device__ __forceinline__ void z_face(C F, C nz, C lo, C hi, bool iz, C & el, C & gl, C & eu, C & gu) {
  const C d = lo - hi;
  if (iz) {
    el = mad(F, d, el);
    gl = mad(-nz, d, gl);
    eu = F * d;
    gu = nz * d;
  } else {
    el = mad(F - nz, d, el);
    eu = (F + nz) * d;
    gu = 0;
  }
}

// The y face r = 0 .. 2 of a pair (below the first line, between the two, above
// the second) of one variable: flux F, diffusion coefficient n, d = value below -
// value above; line r is above the face and line r - 1 below it.
template <class C>
__device__ __forceinline__ void y_face(C F, C n, C d, int r, bool iy, C (&e)[2], C (&g)[2]) {
  if (r > 0) {
    e[r - 1] = mad(F, d, e[r - 1]);
    C & side = iy ? g[r - 1] : e[r - 1];
    side = mad(-n, d, side);
  }
  if (r < 2) {
    e[r] = mad(F, d, e[r]);
    C & side = iy ? g[r] : e[r];
    side = mad(n, d, side);
  }
}

// ------------------------------------------------------------ group A: ux, t
// z faces between the planes V (lower) and N (upper) of both lines: shares of
// the lower cells added to ex, gx (ux) and et, gt (t), those of the upper cells
// returned in x and t (for the next plane)
template <class L, bool TILE, class C, class T, class D>
__device__ __forceinline__ void z_faces_a(const CoefA<C> & q, const CoefZ<C> & z, const View<L, T, TILE> & V,
                                          const View<L, T, TILE> & N, const D & im, C (&ex)[2], C (&gx)[2], C (&et)[2],
                                          C (&gt)[2], Share<C> & x, Share<C> & t) {
#pragma unroll
  for (int l = 0; l < 2; l++) {
    const C w_m = UZ(N, l + 1, -1), w_0 = UZ(N, l + 1, 0);
    z_face(mad(q.zc1, w_m, q.zc2 * w_0), z.nz, UX(V, l + 1, 0), UX(N, l + 1, 0), im.z, ex[l], gx[l], x.e[l], x.g[l]);
    // diffusion_z1 (ux.c:311-332): uz across the radial face, difference of the two z faces
    const C dw = w_0 - w_m;
    ex[l] = mad(q.cz1, dw, ex[l]);
    x.e[l] = mad(-q.cz1, dw, x.e[l]);
    z_face(z.t * w_0, z.kz, TT(V, l + 1, 0), TT(N, l + 1, 0), im.z, et[l], gt[l], t.e[l], t.g[l]);
  }
}

// explicit and implicit sides of ux at face i (src/fluid/predict/ux.c) and t at
// centre i (t.c) of both lines of plane V but for their lower z faces, which e
// and g hold on entry
template <class L, bool TILE, class C, class T, class D>
__device__ __forceinline__ void sides_a(const CoefA<C> & q, const View<L, T, TILE> & V, const D & im, C (&ex)[2],
                                        C (&gx)[2], C (&et)[2], C (&gt)[2]) {
  const C v_m[3] = {UY(V, 1, -1), UY(V, 2, -1), UY(V, 3, -1)};   // uy at rows j, j + 1, j + 2
  const C v_0[3] = {UY(V, 1, 0), UY(V, 2, 0), UY(V, 3, 0)};
  const C u[4] = {UX(V, 0, 0), UX(V, 1, 0), UX(V, 2, 0), UX(V, 3, 0)};
  C up[2];
#pragma unroll
  for (int l = 0; l < 2; l++) {
    // ux has no unknown at i = 1 (face 1 is the wall): its value there is
    // formed from in-bounds shared-memory neighbours and discarded, so the
    // cell stays one branch-free block
    const C u0 = u[l + 1], um = UX(V, l + 1, -1);
    up[l] = UX(V, l + 1, 1);
    const C dm = um - u0, dp = up[l] - u0, a = q.xa2 * u0;
    // advection in x (ux.c:92-121): 1/J (l q_m + c q_0 + u q_p) with c = -l - u as differences from q_0
    C e = mad(mad(q.xa1, um, a), dm, ex[l]);
    e = mad(-mad(q.xa3, up[l], a), dp, e);
    // centrifugal term (:194-226): 1/J hd (uy averaged to the face)^2
    const C sm = v_m[l] + v_m[l + 1], sp = v_0[l] + v_0[l + 1];
    e = mad(q.h1 * sm, sm, e);
    e = mad(q.h2 * sp, sp, e);
    // diffusion_y1 (:266-290) and the uy part of diffusion_a (:344-375) as
    // differences of uy across j, the ux part of diffusion_a
    e = mad(q.cy1, v_m[l + 1] - v_m[l], e);
    e = mad(q.cy2, v_0[l + 1] - v_0[l], e);
    e = mad(q.ca1, um + u0, e);
    e = mad(q.ca2, u0 + up[l], e);
    // diffusion in x
    C & side = im.x ? gx[l] : e;
    side = mad(q.lxl, dm, side);
    side = mad(q.lxu, dp, side);
    ex[l] = e;
    // pressure gradient (:377-394)
    const C dpx = (C)(PP(V, l + 1, 0) - PP(V, l + 1, -1));
    gx[l] = mad(-q.px, dpx, gx[l]);
  }
  // y faces (:123-155) below the first line, between the two and above the second
#pragma unroll
  for (int r = 0; r < 3; r++) {
    y_face(mad(q.yb1, v_m[r], q.yb2 * v_0[r]), q.ly, u[r] - u[r + 1], r, im.y, ex, gx);
  }
  // t (t.c:88-116) with the face velocities
  const C t[4] = {TT(V, 0, 0), TT(V, 1, 0), TT(V, 2, 0), TT(V, 3, 0)};
#pragma unroll
  for (int l = 0; l < 2; l++) {
    const C dm = TT(V, l + 1, -1) - t[l + 1], dp = TT(V, l + 1, 1) - t[l + 1];
    et[l] = mad(q.tx0 * u[l + 1], dm, et[l]);
    et[l] = mad(-q.tx1 * up[l], dp, et[l]);
    C & side = im.x ? gt[l] : et[l];
    side = mad(q.kl, dm, side);
    side = mad(q.ku, dp, side);
  }
#pragma unroll
  for (int r = 0; r < 3; r++) y_face(q.ty * v_0[r], q.ky, t[r] - t[r + 1], r, im.y, et, gt);
}

// ------------------------------------------------------------ group B: uy, uz
template <class L, bool TILE, class C, class T, class D>
__device__ __forceinline__ void z_faces_b(const CoefB<C> & q, const CoefZ<C> & z, const View<L, T, TILE> & V,
                                          const View<L, T, TILE> & N, const D & im, C (&ey)[2], C (&gy)[2], C (&ez)[2],
                                          C (&gz)[2], Share<C> & y, Share<C> & w) {
  const C n[3] = {UZ(N, 0, 0), UZ(N, 1, 0), UZ(N, 2, 0)};   // uz at the face, rows j - 1, j, j + 1
#pragma unroll
  for (int l = 0; l < 2; l++) {
    z_face(z.c * (n[l] + n[l + 1]), z.nz, UY(V, l + 1, 0), UY(N, l + 1, 0), im.z, ey[l], gy[l], y.e[l], y.g[l]);
    // diffusion_z1 (uy.c): uz across j, difference of the two z faces
    const C dn = n[l + 1] - n[l];
    ey[l] = mad(q.yz, dn, ey[l]);
    y.e[l] = mad(-q.yz, dn, y.e[l]);
    // uz's own z faces are the cell centres: the flux is the mean of both planes' uz
    const C lo = UZ(V, l + 1, 0);
    z_face(z.c * (lo + n[l + 1]), C(2) * z.nz, lo, n[l + 1], im.z, ez[l], gz[l], w.e[l], w.g[l]);
  }
}

// explicit and implicit sides of uy (src/fluid/predict/uy.c) and uz (uz.c) at
// centre i of both lines of plane V (M: the plane below)
template <class L, bool TILE, class C, class T, class D>
__device__ __forceinline__ void sides_b(const CoefB<C> & q, const CoefZ<C> & z, const View<L, T, TILE> & V,
                                        const View<L, T, TILE> & M, const D & im, C (&ey)[2], C (&gy)[2], C (&ez)[2],
                                        C (&gz)[2]) {
  const C x0[3] = {UX(V, 0, 0), UX(V, 1, 0), UX(V, 2, 0)}, x1[3] = {UX(V, 0, 1), UX(V, 1, 1), UX(V, 2, 1)};
  const C v[4] = {UY(V, 0, 0), UY(V, 1, 0), UY(V, 2, 0), UY(V, 3, 0)};
  C s[3];   // uy sums across the y faces at rows j - 1/2, j + 1/2, j + 3/2
#pragma unroll
  for (int r = 0; r < 3; r++) s[r] = v[r] + v[r + 1];
#pragma unroll
  for (int l = 0; l < 2; l++) {
    const C v0 = v[l + 1], vm = UY(V, l + 1, -1), vp = UY(V, l + 1, 1);
    const C dm = vm - v0, dp = vp - v0;
    const C wm = x0[l] + x1[l], w0 = x0[l + 1] + x1[l + 1];
    // advection in x (uy.c:93-123)
    C e = mad(q.a1 * (x0[l] + x0[l + 1]), dm, ey[l]);
    e = mad(-q.a2 * (x1[l] + x1[l + 1]), dp, e);
    // advection_1 (:188-223): -1/J hd (uy ux averaged to j -/+ 1/2)
    e = mad(-q.h, mad(s[l], wm, s[l + 1] * w0), e);
    // diffusion_x1 + diffusion_a (lyx at faces i, i+1 and lxy), diffusion_y1 (lyy1 at j-1, j)
    e = mad(q.p1, x0[l + 1] - x0[l], e);
    e = mad(q.p2, x1[l + 1] - x1[l], e);
    e = mad(q.qm, vm, e);
    e = mad(q.q0, v0, e);
    e = mad(q.qp, vp, e);
    e = mad(q.yk, w0 - wm, e);
    const double p0 = PP(V, l + 1, 0);
    const C dpy = (C)(p0 - PP(V, l, 0)), dpz = (C)(p0 - PP(M, l + 1, 0));
    C & side = im.x ? gy[l] : e;
    side = mad(q.lxl, dm, side);
    side = mad(q.lxu, dp, side);
    ey[l] = e;
    gy[l] = mad(-q.py, dpy, gy[l]);
    gz[l] = mad(-z.ih, dpz, gz[l]);
    // uz: advection in x (uz.c:88-118) and diffusion_x1 (lzx at faces i, i+1)
    const C m0 = UX(M, l + 1, 0), m1 = UX(M, l + 1, 1);
    const C z0 = UZ(V, l + 1, 0), zm = UZ(V, l + 1, -1) - z0, zp = UZ(V, l + 1, 1) - z0;
    C f = mad(q.a1 * (m0 + x0[l + 1]), zm, ez[l]);
    f = mad(-q.a2 * (m1 + x1[l + 1]), zp, f);
    f = mad(q.zx1, x1[l + 1] - m1, f);
    f = mad(-q.zx0, x0[l + 1] - m0, f);
    C & zside = im.x ? gz[l] : f;
    zside = mad(q.lxl, zm, zside);
    zside = mad(q.lxu, zp, zside);
    ez[l] = f;
  }
  const C w[4] = {UZ(V, 0, 0), UZ(V, 1, 0), UZ(V, 2, 0), UZ(V, 3, 0)};
#pragma unroll
  for (int r = 0; r < 3; r++) {
    // uy's y faces are the cell centres (:125-151), diffusion 2 nu / hy^2
    y_face(q.b * s[r], C(2) * q.ly, v[r] - v[r + 1], r, im.y, ey, gy);
    // uz's y faces (uz.c:120-150), advected by uy of both planes; diffusion_y1 (lzy at j, j+1)
    const C mv = UY(M, r + 1, 0);
    y_face(q.b * (mv + v[r + 1]), q.ly, w[r] - w[r + 1], r, im.y, ez, gz);
    const C dv = v[r + 1] - mv;
    if (r > 0) ez[r - 1] = mad(q.yz, dv, ez[r - 1]);
    if (r < 2) ez[r] = mad(-q.yz, dv, ez[r]);
  }
}
#undef UX
#undef UY
#undef UZ
#undef TT
#undef PP

template <int E>
__device__ __forceinline__ int spad(int e) { return e + e / E; }

// Radial Thomas solves of LN lines by one warp (src/tdm.c:24-48): lane t owns
// elements tE .. tE+E-1 of each. With the pivots 1 / w the sweeps are
//   p_m = r_m + f_m p_{m-1}, f_m = -l_m w_{m-1};  s_m = p_m + g_m s_{m+1}, g_m = -u_m w_{m+1};  x_m = w_m s_m,
// one multiply-add an element. A lane first forms its chunk's last value with
// nothing entering, a 5-level shuffle scan turns those into the values entering
// the chunks, and the lane runs its chunk again from there. The products of f
// (and g) that the scan levels multiply by do not depend on the right-hand side:
// xfactor_kernel tabulates them per lane (scan rows 0-4 forward, 5-9 backward),
// zero where a level has no source lane, so a level is one shuffle and one
// multiply-add. The factors of a lane stay in registers for all its lines; several
// lines at a time (stride doubles apart) hide the chains' and the shuffles' latency.
// Elements from n on have f = g = w = 0. Per plane of two 256-point lines: 1.55k
// cycles, against 4.2k with the factor rows read and multiplied out for each line.
// SINGLE (FP32-storage contexts) keeps the former order of roundings: r_m w_m
// first, f_m = -w_m l_m and g_m = -v_m with the rows' l, w, v (XFactors::single).
template <int E, bool SINGLE>
struct LineFactors {
  double f[E], g[E], w[E], up[5], down[5];
  // rows are interleaved: element lane E + m at m 32 + lane
  __device__ __forceinline__ void load(const XFactors & xf, int rk, int v, int lane) {
    const size_t o = (size_t)(rk * 4 + v) * xf.stride + lane;
    const double * sc = xf.scan + (size_t)(rk * 4 + v) * XSCAN_ROWS * 32 + lane;
#pragma unroll
    for (int m = 0; m < E; m++) {
      f[m] = LD(xf.f + o + m * 32);
      g[m] = LD(xf.g + o + m * 32);
      w[m] = LD(xf.w + o + m * 32);
      if (SINGLE) {
        f[m] = __dmul_rn(-w[m], f[m]);
        g[m] = -g[m];
      }
    }
#pragma unroll
    for (int q = 0; q < 5; q++) {
      up[q] = LD(sc + q * 32);
      down[q] = LD(sc + (5 + q) * 32);
    }
  }
};
template <int E, int LN, bool SINGLE>
__device__ __forceinline__ void solve_lines(double * sb, int stride, const LineFactors<E, SINGLE> & x, int lane) {
  double r[LN][E], B[LN];
  sb += spad<E>(lane * E);   // the lane's E elements are consecutive
#pragma unroll
  for (int n = 0; n < LN; n++)
#pragma unroll
    for (int m = 0; m < E; m++) r[n][m] = SINGLE ? __dmul_rn(x.w[m], sb[n * stride + m]) : sb[n * stride + m];
#pragma unroll
  for (int n = 0; n < LN; n++) {
    B[n] = r[n][0];
#pragma unroll
    for (int m = 1; m < E; m++) B[n] = fma(x.f[m], B[n], r[n][m]);
  }
#pragma unroll
  for (int q = 0; q < 5; q++)
#pragma unroll
    for (int n = 0; n < LN; n++) B[n] = fma(x.up[q], __shfl_up_sync(0xffffffffu, B[n], 1 << q), B[n]);
#pragma unroll
  for (int n = 0; n < LN; n++) {
    double p = __shfl_up_sync(0xffffffffu, B[n], 1);   // lane 0: f[0] = 0
#pragma unroll
    for (int m = 0; m < E; m++) p = r[n][m] = fma(x.f[m], p, r[n][m]);
    B[n] = r[n][E - 1];
#pragma unroll
    for (int m = E - 2; m >= 0; m--) B[n] = fma(x.g[m], B[n], r[n][m]);
  }
#pragma unroll
  for (int q = 0; q < 5; q++)
#pragma unroll
    for (int n = 0; n < LN; n++) B[n] = fma(x.down[q], __shfl_down_sync(0xffffffffu, B[n], 1 << q), B[n]);
#pragma unroll
  for (int n = 0; n < LN; n++) {
    double p = __shfl_down_sync(0xffffffffu, B[n], 1);   // lane 31: g of the last element is 0
#pragma unroll
    for (int m = E - 1; m >= 0; m--) {
      p = fma(x.g[m], p, r[n][m]);
      sb[n * stride + m] = SINGLE ? p : x.w[m] * p;
    }
  }
}

// the slot of plane kp and the parity of its fill (planes k0 - 1 .. k1 pass
// through the slots in turn)
template <class L>
__device__ __forceinline__ int slot_of(int kp, int k0) { return (kp - k0 + 1) % L::NSLOT; }
template <class L>
__device__ __forceinline__ unsigned fill_of(int kp, int k0) { return ((kp - k0 + 1) / L::NSLOT) & 1u; }

// one CTA's share of the grid: lines j0 .. j0 + nl - 1, planes k0 .. k1 - 1,
// radial indices ib + 1 .. ib + NT
struct Box {
  int j0, nl, k0, k1, ib;
};

// ------------------------------------------------------------ copies
// Solve warp v copies its variable's rows of each plane (planes k0 - 1 .. k1)
// into the ring, warp VUX those of p too, and its variable's old source terms
// (planes k0 .. k1 - 1) into their buffers. A lane owns one copy of every plane:
// lane 0 the rows of the warp's field, lane 1 those of p, or (TILE) one row each,
// from centre index ib and, in double, from ux element ib - 2 on; addresses
// advance by a constant from plane to plane. The consumers' reads of a slot or
// buffer are ordered before the copies into it by the barrier waited for.
template <class L, class T, bool TILE>
struct Copies {
  const char * src;
  size_t step;                  // bytes from plane to plane
  unsigned bytes, off, total;   // of this copy, within the slot; of the warp's copies of a plane
  const T * old;
  size_t old_step;
  unsigned old_bytes;
  int next, next_old;           // next planes to issue

  __device__ __forceinline__ void begin(const Args<T> & A, const Box & x, int v) {
    constexpr bool D64 = L::D64;
    const int q = threadIdx.x & 31, nx = A.g.nx, nf = TILE ? x.nl + 2 : 1;
    const int f = q < nf ? (v == VT ? 3 : v) : 4, r = q < nf ? q : q - nf;   // field 0 .. 3 (ux, uy, uz, t) or 4 (p); row
    const bool use = f < 4 || (v == VUX && r < (TILE ? x.nl + 1 : 1));
    const int rows = TILE ? 1 : f == 4 ? x.nl + 1 : x.nl + 2;
    const size_t es = f == 4 ? sizeof(double) : sizeof(T), al = 16 / es;
    const size_t len = f == 4 || (D64 && f != 0) ? (size_t)nx + 2 : D64 ? (size_t)nx + 1 : (size_t)pitch32(nx);
    const size_t e0 = !TILE ? 0 : f == 0 && D64 ? (x.ib > 0 ? x.ib - 2 : 0) : x.ib;
    const size_t want = f == 0 && D64 ? L::NT + 3 : L::NT + 2;
    const size_t n = TILE ? (len - e0 > want ? want : len - e0) : len * rows;
    const size_t sj = (size_t)A.g.ny + 2;
    const size_t s = len * ((size_t)(x.j0 - 1 + r) + sj * (size_t)(x.k0 - 1)) + e0;
    // widened to 16-byte bounds: at most one double before and after
    const size_t a = s & ~(al - 1), b = (s + n + al - 1) & ~(al - 1);
    const char * base = reinterpret_cast<const char *>(
        f == 0 ? (const void *)A.in.ux : f == 1 ? (const void *)A.in.uy : f == 2 ? (const void *)A.in.uz
        : f == 3 ? (const void *)A.in.t : (const void *)A.in.p);
    src = base + a * es;
    step = len * sj * es;
    bytes = use ? (unsigned)((b - a) * es) : 0u;
    // a tile's face e0 + 1 sits at cell offset e0 + 1 - ib
    const int odd = nx & 1, rs = L::RL + (D64 || f == 4 ? odd : 0);
    const int o = f == 4 ? r * rs
                         : L::FB(f) + r * rs + (TILE && D64 && f == 0 ? (int)e0 + 1 - x.ib + ux_shift<T, TILE>(r) : 0);
    off = (unsigned)((f == 4 ? L::POFF : 0) + (size_t)o * es - (s - a) * es);
    total = bytes;
    for (int d = 16; d > 0; d >>= 1) total += __shfl_xor_sync(0xffffffffu, total, d);
    total += A.lost;
    next = x.k0 - 1;
    // the CTA's lines of a variable are consecutive in the packed layout; an even
    // number of lines before them starts them on a 16-byte boundary
    const int li = D64 ? (v == VUX ? nx - 1 : nx) : spitch32(nx);
    old = A.ss.old_[v] + pidx(li, A.g.ny, 0, x.j0, x.k0);
    old_step = (size_t)li * A.g.ny;
    old_bytes = (unsigned)((size_t)x.nl * li * sizeof(T));
    next_old = TILE || A.rkstep == 0 ? x.k1 : x.k0;
  }
  // the next plane into its slot, once the plane before it there is released
  __device__ __forceinline__ void plane(const Box & x, char * ring, const Bars<L> & bars, volatile int * abort_flag) {
    const int m = next - x.k0 + 1, sl = m % L::NSLOT;
    if (next > x.k1) return;
    if (m >= L::NSLOT) await(bars.empty(sl), (unsigned)(m / L::NSLOT - 1) & 1u, abort_flag);
    if (__any_sync(0xffffffffu, *abort_flag != 0)) return;
    if ((threadIdx.x & 31) == 0) mbar_expect_tx(bars.full(sl), total);
    __syncwarp();
    if (bytes) bulk_g2s(ring + (size_t)sl * L::SLOT + off, src, bytes, bars.full(sl));
    src += step;
    next++;
  }
  // the next plane's old terms; the fields are done with the buffer
  __device__ __forceinline__ void old_terms(const Box & x, T * olds, int v, const Bars<L> & bars,
                                            volatile int * abort_flag) {
    if (next_old >= x.k1 || *abort_flag) return;
    const int q = (next_old - x.k0) & 1;
    if ((threadIdx.x & 31) == 0) {
      mbar_expect_tx(bars.olds(q), old_bytes);
      bulk_g2s(olds + (size_t)(q * 4 + v) * L::JT * L::OL, old, old_bytes, bars.olds(q));
    }
    old += old_step;
    next_old++;
  }
  // No copy outlives the CTA: wait, one limit for all of them, for the latest fill of
  // each slot and buffer (on the ordinary path the consumers wait for them too).
  __device__ __forceinline__ void drain(const Args<T> & A, const Box & x, const Bars<L> & bars) {
    const long long t0 = clock64();
    auto settle = [&](unsigned long long * bar, unsigned parity) {
      while (!mbar_try_wait(bar, parity))
        if (clock64() - t0 > kWaitCycles) return;
    };
    for (int kp = next - L::NSLOT > x.k0 - 1 ? next - L::NSLOT : x.k0 - 1; kp < next; kp++)
      settle(bars.full(slot_of<L>(kp, x.k0)), fill_of<L>(kp, x.k0));
    if constexpr (!TILE)
      for (int ko = next_old - 2 > x.k0 ? next_old - 2 : x.k0; ko < next_old && A.rkstep != 0; ko++)
        settle(bars.olds((ko - x.k0) & 1), (unsigned)((ko - x.k0) / 2) & 1u);
  }
};

// ------------------------------------------------------------ field warps
// One group's state in a thread: radial index i = ib + is of line pair pr.
template <class L, int GRP, int IMPL, class T, bool TILE>
struct Group {
  static constexpr bool D64 = L::D64;
  static constexpr int VA = GRP == 0 ? VUX : VUY, VB = GRP == 0 ? VT : VUZ;
  using C = T;
  typename std::conditional<GRP == 0, CoefA<C>, CoefB<C>>::type q;
  Share<C> ua, ub;           // the lower z faces' shares of the next plane to form
  T * na, * nb;              // new source terms of the pair's first line, next plane
  const T * ga, * gb;        // tiles: old source terms (read from global memory)
  const double * fa, * fb;   // closure forcing (double, same packed layout: FP64 storage)
  const T * oa, * ob;        // old source terms in shared memory
  double * st;
  int la, lc, pa, pb;
  bool act, acta;

  __device__ __forceinline__ void begin(const Args<T> & A, const Box & x, double * stage, const T * olds, int pr,
                                        int is) {
    const int nx = A.g.nx, ny = A.g.ny, i = x.ib + is;
    act = i <= nx && 2 * pr < x.nl;
    acta = act && (GRP == 1 || i >= 2);   // ux has no unknown at i = 1
    load_coefs(q, A.cf, i <= nx ? i : 1, A.nu, A.kappa);
    const int lf = D64 ? nx - 1 : spitch32(nx);   // source-term lines (sline)
    lc = D64 ? nx : spitch32(nx);
    la = GRP == 0 ? lf : lc;
    const int ia = GRP == 0 ? i - 2 : i - 1;
    const size_t qa = pidx(la, ny, ia, x.j0 + 2 * pr, x.k0), qb = pidx(lc, ny, i - 1, x.j0 + 2 * pr, x.k0);
    na = A.ss.new_[VA] + qa;
    nb = A.ss.new_[VB] + qb;
    ga = TILE && A.rkstep != 0 ? A.ss.old_[VA] + qa : nullptr;
    gb = TILE && A.rkstep != 0 ? A.ss.old_[VB] + qb : nullptr;
    if constexpr (forced(IMPL)) {
      fa = A.ss.frc[VA] + qa;
      fb = GRP == 1 ? A.ss.frc[VB] + qb : nullptr;
    }
    // at i = 1 the old ux term read is the word before the line (discarded)
    oa = olds + (size_t)VA * L::JT * L::OL + 2 * pr * la + ia;
    ob = olds + (size_t)VB * L::JT * L::OL + 2 * pr * lc + i - 1;
    st = stage + (size_t)(2 * pr * 4) * L::SL;
    // staging positions: unknown 0 of ux is face 2; tiles, which are not solved here, count from face ib + 1
    pa = spad<L::E>(GRP == 0 && !TILE ? is - 2 : is - 1);
    pb = spad<L::E>(is - 1);
  }
  // the z faces below the first plane V (M: the plane under it)
  __device__ __forceinline__ void below(const CoefZ<C> & z, const View<L, T, TILE> & M, const View<L, T, TILE> & V,
                                        const Dirs<IMPL> & im) {
    C e0[2] = {0, 0}, g0[2] = {0, 0}, e1[2] = {0, 0}, g1[2] = {0, 0};
    if constexpr (GRP == 0) z_faces_a<L, TILE>(q, z, M, V, im, e0, g0, e1, g1, ua, ub);
    else z_faces_b<L, TILE>(q, z, M, V, im, e0, g0, e1, g1, ua, ub);
  }
  // plane V between M and N: new source terms out, increments into staging
  // buffer b; ca, cb, cg = alpha dt, beta dt, gamma dt
  __device__ __forceinline__ void plane(const Args<T> & A, const CoefZ<C> & z, const View<L, T, TILE> & M,
                                        const View<L, T, TILE> & V, const View<L, T, TILE> & N, const Dirs<IMPL> & im,
                                        const Bars<L> & bars, volatile int * abort_flag, int step, C ca, C cb, C cg) {
    const size_t sa = (size_t)la * A.g.ny, sb = (size_t)lc * A.g.ny;   // plane strides
    T o_a[2] = {0, 0}, o_b[2] = {0, 0};   // tiles read the old terms ahead of their use
    if (TILE && A.rkstep != 0) {
#pragma unroll
      for (int l = 0; l < 2; l++) {
        if (acta) o_a[l] = ga[(size_t)l * la + step * sa];
        if (act) o_b[l] = gb[(size_t)l * lc + step * sb];
      }
    }
    C ea[2], g_a[2], eb[2], g_b[2];
#pragma unroll
    for (int l = 0; l < 2; l++) { ea[l] = ua.e[l]; g_a[l] = ua.g[l]; eb[l] = ub.e[l]; g_b[l] = ub.g[l]; }
    if constexpr (GRP == 0) {
      z_faces_a<L, TILE>(q, z, V, N, im, ea, g_a, eb, g_b, ua, ub);
      sides_a<L, TILE>(q, V, im, ea, g_a, eb, g_b);
    } else {
      z_faces_b<L, TILE>(q, z, V, N, im, ea, g_a, eb, g_b, ua, ub);
      sides_b<L, TILE>(q, z, V, M, im, ea, g_a, eb, g_b);
    }
    if constexpr (forced(IMPL)) {
#pragma unroll
      for (int l = 0; l < 2; l++) {
        if (acta) ea[l] += (C)fa[(size_t)l * la + step * sa];
        if (GRP == 1 && act) eb[l] += (C)fb[(size_t)l * lc + step * sb];
      }
      if (step + 1 < A.KC) {   // the next plane's forces into the L1 (held in registers they spill)
#pragma unroll
        for (int l = 0; l < 2; l++) {
          if (acta) prefetch_l1(fa + (size_t)l * la + (step + 1) * sa);
          if (GRP == 1 && act) prefetch_l1(fb + (size_t)l * lc + (step + 1) * sb);
        }
      }
    }
    if (!TILE && A.rkstep != 0) {
      const int buf = (step & 1) * 4 * L::JT * L::OL;
      await(bars.olds(step & 1), (unsigned)(step >> 1) & 1u, abort_flag);
#pragma unroll
      for (int l = 0; l < 2; l++) {
        o_a[l] = oa[buf + l * la];
        o_b[l] = ob[buf + l * lc];
      }
    }
    double * sd = st + (size_t)(step & 1) * L::JT * 4 * L::SL;
#pragma unroll
    for (int l = 0; l < 2; l++) {
      C da = mad(ca, ea[l], cg * g_a[l]), db = mad(ca, eb[l], cg * g_b[l]);
      if (A.rkstep != 0) {
        da = mad(cb, (C)o_a[l], da);
        db = mad(cb, (C)o_b[l], db);
      }
      if (acta) {
        na[l * la] = (T)ea[l];
        sd[(l * 4 + VA) * L::SL + pa] = (double)da;
      }
      if (act) {
        nb[l * lc] = (T)eb[l];
        sd[(l * 4 + VB) * L::SL + pb] = (double)db;
      }
    }
    na += sa;
    nb += sb;
  }
};
struct NoGroup {
  template <class... X> __device__ __forceinline__ void begin(X &&...) {}
  template <class... X> __device__ __forceinline__ void below(X &&...) {}
  template <class... X> __device__ __forceinline__ void plane(X &&...) {}
};

// wg: the warp among those of its groups (GA: forms ux and t, GB: uy and uz)
template <class L, bool GA, bool GB, int IMPL, class T, bool TILE>
__device__ __forceinline__ void fields(const Args<T> & A, const Box & x, char * ring, double * stage, const T * olds,
                                       const Bars<L> & bars, volatile int * abort_flag, double dt, int wg) {
  using C = T;
  constexpr bool D64 = L::D64;
  const int nx = A.g.nx, lane = threadIdx.x & 31;
  const int pr = L::PAIRS == 1 ? 0 : wg / L::NW;
  const int is = (L::PAIRS == 1 ? wg : wg % L::NW) * 32 + lane + 1;   // i - ib
  const Dirs<IMPL> im(A.bc);
  const double ihz = A.cf.inv_hz;
  const CoefZ<C> z{(C)(A.nu * A.cf.lz_l), (C)(A.kappa * A.cf.lz_l), (C)(0.5 * ihz), (C)(0.25 * ihz), (C)ihz};
  const int rk = A.rkstep;
  const C ca = (C)(rk_alpha(rk) * dt), cb = (C)(rk_beta(rk) * dt), cg = (C)(rk_gamma(rk) * dt);
  typename std::conditional<GA, Group<L, 0, IMPL, T, TILE>, NoGroup>::type ga;
  typename std::conditional<GB, Group<L, 1, IMPL, T, TILE>, NoGroup>::type gb;
  ga.begin(A, x, stage, olds, pr, is);
  gb.begin(A, x, stage, olds, pr, is);
  const int rs = TILE ? L::RL + (D64 ? nx & 1 : 0) : D64 ? nx + 2 : pitch32(nx);
  const int ps = TILE ? L::RL + (nx & 1) : nx + 2;
  auto view = [&](int kp) {
    const char * s = ring + (size_t)slot_of<L>(kp, x.k0) * L::SLOT;
    View<L, T, TILE> V;
    V.s = rs;
    V.sp = ps;
    V.c = reinterpret_cast<const T *>(s) + 2 * pr * rs + is;
    V.f = V.c + (D64 ? (TILE ? 2 : -2) * pr : 0);
    V.p = reinterpret_cast<const double *>(s + L::POFF) + 2 * pr * ps + is;
    return V;
  };
  await(bars.full(slot_of<L>(x.k0 - 1, x.k0)), 0, abort_flag);
  await(bars.full(slot_of<L>(x.k0, x.k0)), 0, abort_flag);
  View<L, T, TILE> M = view(x.k0 - 1), V = view(x.k0);
  ga.below(z, M, V, im);
  gb.below(z, M, V, im);
  for (int k = x.k0; k < x.k1; k++) {
    const int step = k - x.k0, b = step & 1;
    await(bars.full(slot_of<L>(k + 1, x.k0)), fill_of<L>(k + 1, x.k0), abort_flag);
    if (step >= 2) await(bars.unstaged(b), (unsigned)((step >> 1) - 1) & 1u, abort_flag);
    const View<L, T, TILE> N = view(k + 1);
    ga.plane(A, z, M, V, N, im, bars, abort_flag, step, ca, cb, cg);
    gb.plane(A, z, M, V, N, im, bars, abort_flag, step, ca, cb, cg);
    // this warp is done with plane k - 1 and with the old terms of plane k, and
    // its increments are staged
    __syncwarp();
    if (lane == 0) {
      mbar_arrive(bars.staged(b));
      mbar_arrive(bars.empty(slot_of<L>(k - 1, x.k0)));
    }
    M = V;
    V = N;
  }
}

// ------------------------------------------------------------ solve warps
// Variable v of every line of the CTA, plane after plane: radial solve in the
// staging lines (where x is implicit), then u + delta with walls and images,
// or the increments themselves (line solves in y, z or of tiled lines follow).
template <class L, int IMPL, class T, bool TILE>
__device__ __forceinline__ void solves(const Args<T> & A, const Box & x, char * ring, double * stage, T * olds,
                                       const Bars<L> & bars, volatile int * abort_flag, int v) {
  constexpr int E = L::E;
  const Geo & g = A.g;
  const int nx = g.nx, ny = g.ny, nz = g.nz, lane = threadIdx.x & 31;
  Copies<L, T, TILE> copies;
  copies.begin(A, x, v);
  for (int s = 0; s < L::NSLOT; s++) copies.plane(x, ring, bars, abort_flag);
  copies.old_terms(x, olds, v, bars, abort_flag);
  copies.old_terms(x, olds, v, bars, abort_flag);
  const Dirs<IMPL> im(A.bc);
  const bool solve_x = !TILE && im.x;
  LineFactors<E, sizeof(T) == 4> factors;
  if (solve_x) factors.load(A.xf, A.rkstep, v, lane);
  const int i0 = v == VUX ? 2 : 1;              // radial index of unknown 0
  const int n = v == VUX ? nx - 1 : nx;         // unknowns of a line
  T * out = v == VUX ? A.out.ux : v == VUY ? A.out.uy : v == VUZ ? A.out.uz : A.out.t;
  const int row = v == VUX ? srow_f<T>(g) : srow_c<T>(g);
  const T wm = (T)(v == VUY ? A.bc.uy_xm : v == VT ? A.bc.t_xm : 0.);
  const T wp = (T)(v == VUY ? A.bc.uy_xp : v == VT ? A.bc.t_xp : 0.);
  // radial index 1 of line j0, plane k0 (ux in double: element 0 of its row)
  T * o0 = out + (size_t)row * ((size_t)x.j0 + (size_t)(ny + 2) * x.k0) + (v == VUX && L::D64 ? 0 : 1);
  const size_t oplane = (size_t)row * (ny + 2);
  // current values in the ring slot: unknown 0 of row j0 (not used by tiles)
  const int rs = (L::D64 ? nx + 2 : pitch32(nx)) - (L::D64 && v == VUX ? 1 : 0);
  const int u0 = L::FB(v == VT ? 3 : v) + rs + (v == VUX && !L::D64 ? 2 : 1);
  if (lane == 0) mbar_arrive(bars.empty(slot_of<L>(x.k0 - 1, x.k0)));   // the halo plane: nothing to solve
  for (int k = x.k0; k < x.k1; k++, o0 += oplane) {
    const int step = k - x.k0, b = step & 1;
    await(bars.full(slot_of<L>(k, x.k0)), fill_of<L>(k, x.k0), abort_flag);
    await(bars.staged(b), (unsigned)(step >> 1) & 1u, abort_flag);
    // the fields are done with plane k: refill the slot of k - 1, the old terms of k
    copies.plane(x, ring, bars, abort_flag);
    copies.old_terms(x, olds, v, bars, abort_flag);
    const bool skip = *abort_flag != 0;
    double * sd = stage + ((size_t)b * L::JT * 4 + v) * L::SL;
    const T * us = reinterpret_cast<const T *>(ring + (size_t)slot_of<L>(k, x.k0) * L::SLOT) + u0;
    // all lines of the variable at once (those past ny in the last CTA are zero)
    if (solve_x) {
      solve_lines<E, L::JT, sizeof(T) == 4>(sd, 4 * L::SL, factors, lane);
      __syncwarp();
    }
#pragma unroll 1
    for (int jl = 0; jl < x.nl && !skip; jl += 2) {
      const double * sb[2] = {sd + jl * 4 * L::SL, sd + (jl + 1) * 4 * L::SL};
      if (A.mode == PREDICT_DELTA) {
#pragma unroll
        for (int m = 0; m < 2; m++) {
          double * d = A.ds.d[v] + pidx(n, ny, 0, x.j0 + jl + m, k);
          if (TILE) {   // element e is radial index ib + 1 + e
            const int m0 = x.ib + 1 - i0, cnt = nx - x.ib < L::NT ? nx - x.ib : L::NT;
            for (int e = lane; e < cnt; e += 32)
              if (m0 + e >= 0) d[m0 + e] = sb[m][spad<E>(e)];
          } else {
            for (int e = lane; e < n; e += 32) d[e] = sb[m][spad<E>(e)];
          }
        }
        continue;
      }
      // u + delta of both lines, lanes along the line
#pragma unroll
      for (int m = 0; m < 2; m++) {
        const T * u = us + (jl + m) * rs;
        T * d = o0 + (size_t)(jl + m) * row;
        T val[E];
#pragma unroll
        for (int c = 0; c < E; c++) {
          const int e = c * 32 + lane;
          val[c] = (T)((double)u[e] + sb[m][spad<E>(e)]);
        }
        auto put = [&](T * r) {
#pragma unroll
          for (int c = 0; c < E; c++)
            if (c * 32 + lane < n) r[c * 32 + lane + i0 - 1] = val[c];
          if (lane == 0) {
            r[v == VUX ? 0 : -1] = wm;
            r[nx] = wp;
          }
        };
        put(d);
        const int j = x.j0 + jl + m;
        if (j == 1 || j == ny || k == 1 || k == nz)
          for_images(j, k, ny, nz, [&](int jj, int kk) {
            put(d + (ptrdiff_t)row * ((ptrdiff_t)(jj - j) + (ptrdiff_t)(ny + 2) * (kk - k)));
          });
      }
    }
    __syncwarp();
    if (lane == 0) {
      mbar_arrive(bars.unstaged(b));
      mbar_arrive(bars.empty(slot_of<L>(k, x.k0)));
    }
  }
  copies.drain(A, x, bars);
}

// registers per thread of this warpgroup from now on (0: as launched)
template <int R, int LAUNCH>
__device__ __forceinline__ void set_regs() {
  if constexpr (R > LAUNCH) asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(R));
  else if constexpr (R > 0) asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(R));
}

template <int NW, int PAIRS, int NG, int IMPL, class T, bool TILE>
__global__ void __launch_bounds__(Layout<NW, PAIRS, NG, T>::THREADS, 1)
predict_kernel(Args<T> A, const double * __restrict__ dtp) {
  using L = Layout<NW, PAIRS, NG, T>;
  extern __shared__ __align__(16) double sm[];
  char * ring = reinterpret_cast<char *>(sm);
  double * stage = reinterpret_cast<double *>(ring + L::STAGE);
  T * olds = reinterpret_cast<T *>(ring + L::OLDS);
  const Bars<L> bars{reinterpret_cast<unsigned long long *>(ring + L::BAR)};
  volatile int * abort_flag = reinterpret_cast<volatile int *>(bars.b + L::NBAR);
  const int tx = threadIdx.x, warp = tx >> 5;
  const int njg = (A.g.ny + L::JT - 1) / L::JT;
  const int ntile = TILE ? (A.g.nx + L::NT - 1) / L::NT : 1;
  const unsigned bl = TILE ? blockIdx.x / ntile : blockIdx.x;
  Box x;
  x.ib = TILE ? (int)(blockIdx.x % ntile) * L::NT : 0;
  x.j0 = (int)(bl % njg) * L::JT + 1;   // odd
  x.nl = A.g.ny - x.j0 + 1 < L::JT ? A.g.ny - x.j0 + 1 : L::JT;   // even
  x.k0 = (int)(bl / njg) * A.KC + 1;
  x.k1 = x.k0 + A.KC;   // planes k0 .. k1-1 are computed; k0-1 .. k1 are read
  if (tx == 0) {
    for (int s = 0; s < L::NSLOT; s++) {
      mbar_init(bars.full(s), L::NSW);
      mbar_init(bars.empty(s), L::NFW + L::NSW);
    }
    for (int q = 0; q < 2; q++) {
      mbar_init(bars.staged(q), L::NFW);
      mbar_init(bars.unstaged(q), L::NSW);
      mbar_init(bars.olds(q), L::NSW);
    }
    *abort_flag = 0;
    fence_mbar_init();
  }
  // staging lines are zero past each line's unknowns for the whole march
  for (int e = tx; e < 2 * L::JT * 4 * L::SL; e += blockDim.x) stage[e] = 0.;
  __syncthreads();
  if (warp < L::NFW) {
    set_regs<L::REGS_FIELD, L::REGS>();
    if constexpr (NG == 1)
      fields<L, true, true, IMPL, T, TILE>(A, x, ring, stage, olds, bars, abort_flag, *dtp, warp);
    else if (warp < L::NFW / 2)
      fields<L, true, false, IMPL, T, TILE>(A, x, ring, stage, olds, bars, abort_flag, *dtp, warp);
    else
      fields<L, false, true, IMPL, T, TILE>(A, x, ring, stage, olds, bars, abort_flag, *dtp, warp - L::NFW / 2);
  } else {
    set_regs<L::REGS_SOLVE, L::REGS>();
    solves<L, IMPL, T, TILE>(A, x, ring, stage, olds, bars, abort_flag, warp - L::NFW);
  }
  __syncthreads();
  if (tx == 0 && *abort_flag) atomicOr(A.status, ST_TIMEOUT);
}

}  // namespace march
}  // namespace tcgpu
