// The right-hand sides and increments of the marching predict kernel in FP32-storage
// contexts: float arithmetic on the float fields (differences of the double p rounded
// once); the increments are widened for the radial solves and the update, which are double. The order of every
// rounding is part of the mode's results (a single-precision state has no room
// below its rounding: another order of the same sums changes the last bit of
// stored values, and through them the time step), so each cell keeps the plain
// per-cell form of its terms instead of the shared faces of tc_march.cuh.
// What bounds it, and the roles: tc_march.cuh. Per launch at 128 x 512 x 256: 1.22 ms
// in a kernel of its own whose field warps waited for the solutions, 0.50 here.
#pragma once
#include "tc_march.cuh"

namespace tcgpu {
namespace march {

struct CoefA32 {
  float xa1, xa2, xa3, yb1, yb2, zc1, zc2, h1, h2;   // ux advection, centrifugal term
  float lxl, lxu, ly;                                // ux Laplacian, x and y (carry 2 nu, nu)
  float cy1, cy2, ca1, ca2, cz1, px;                 // ux cross diffusion (carry nu), pressure gradient
  float tx0, tx1, ty, tz;                            // t advection
  float clxl, clxu, cly;                             // centred Laplacian, x and y (carry nu; t: times kappa / nu)
};
struct CoefB32 {
  float a1, a2, b, c, h;                             // uy / uz advection
  float lxl, lxu, ly;                                // centred Laplacian, x and y (carry nu)
  float p1, p2, qm, q0, qp, yk, yz, py;              // uy cross diffusion (carry nu), pressure gradient
  float zx0, zx1, zy;                                // uz cross diffusion (carry nu)
};
struct CoefZ32 {
  float l, c, u, ihz;                                // z Laplacian, 1 / hz
};
__device__ __forceinline__ void load_coefs32(CoefA32 & q, const Coefs & cf, int i, double nu_) {
  const double * __restrict__ b = cf.tab + i;
  const float nu = (float)nu_, n2 = (float)(2. * nu_);
#define CF(T) (float)LD(b + (T) * CSTRIDE)
  q.xa1 = CF(P_XA1); q.xa2 = CF(P_XA2); q.xa3 = CF(P_XA3); q.yb1 = CF(P_YB1); q.yb2 = CF(P_YB2);
  q.zc1 = CF(P_ZC1); q.zc2 = CF(P_ZC2); q.h1 = CF(P_H1); q.h2 = CF(P_H2);
  q.lxl = CF(F_LXL) * n2; q.lxu = CF(F_LXU) * n2; q.ly = CF(F_LYL) * nu;
  q.cy1 = CF(P_CY1) * nu; q.cy2 = CF(P_CY2) * nu; q.ca1 = CF(P_CA1) * nu; q.ca2 = CF(P_CA2) * nu;
  q.cz1 = CF(P_CZ1) * nu; q.px = CF(C_INVHXXF);
  q.tx0 = CF(P_TX0); q.tx1 = CF(P_TX1); q.ty = CF(P_TY); q.tz = CF(P_TZ);
  q.clxl = CF(C_LXL) * nu; q.clxu = CF(C_LXU) * nu; q.cly = CF(C_LYL) * nu;
}
__device__ __forceinline__ void load_coefs32(CoefB32 & q, const Coefs & cf, int i, double nu_) {
  const double * __restrict__ b = cf.tab + i;
  const float nu = (float)nu_;
  q.a1 = CF(P_UA1); q.a2 = CF(P_UA2); q.b = CF(P_UB); q.c = CF(P_UC); q.h = CF(P_UH);
  q.lxl = CF(C_LXL) * nu; q.lxu = CF(C_LXU) * nu; q.ly = CF(C_LYL) * nu;
  q.p1 = CF(P_P1) * nu; q.p2 = CF(P_P2) * nu; q.qm = CF(P_QM) * nu; q.q0 = CF(P_Q0) * nu; q.qp = CF(P_QP) * nu;
  q.yk = CF(P_YK) * nu; q.yz = CF(P_YZ) * nu; q.py = CF(C_INVHYXC);
  q.zx0 = CF(P_ZX0) * nu; q.zx1 = CF(P_ZX1) * nu; q.zy = CF(P_ZY) * nu;
#undef CF
}

// element (DI, DJ) from the cell of line JL of the pair: planes k (V), k + 1 (N), k - 1 (M)
#define ROW_(W, F, DJ) ((JL + 1 + (DJ)) * (W).s + L::FB(F))
#define UX(DI, DJ) V.f[ROW_(V, 0, DJ) + (DI)]
#define UY(DI, DJ) V.c[ROW_(V, 1, DJ) + (DI)]
#define UZ(DI, DJ) V.c[ROW_(V, 2, DJ) + (DI)]
#define TT(DI, DJ) V.c[ROW_(V, 3, DJ) + (DI)]
#define PP(DI, DJ) V.p[(JL + 1 + (DJ)) * V.sp + (DI)]
#define NUX(DI) N.f[ROW_(N, 0, 0) + (DI)]
#define NUY(DI) N.c[ROW_(N, 1, 0) + (DI)]
#define NUZ(DI, DJ) N.c[ROW_(N, 2, DJ) + (DI)]
#define NTT(DI) N.c[ROW_(N, 3, 0) + (DI)]
#define MUX(DI) M.f[ROW_(M, 0, 0) + (DI)]
#define MUY(DJ) M.c[ROW_(M, 1, DJ)]
#define MUZ() M.c[ROW_(M, 2, 0)]
#define MTT() M.c[ROW_(M, 3, 0)]
#define MPP() M.p[(JL + 1) * M.sp]
// diffusion in direction D goes to the implicit part when D is implicit
#define ROUTE(D, V_) do { if (D) gi += (V_); else e += (V_); } while (0)

// ux at face i (src/fluid/predict/ux.c) and t at centre i (t.c) of line JL: new
// source terms and increments
template <class L, int JL, bool TILE, class D>
__device__ __forceinline__ void cell32(const CoefA32 & q, const View<L, float, TILE> & M, const View<L, float, TILE> & V,
                                       const View<L, float, TILE> & N, const D & im, const CoefZ32 & lz, float nu,
                                       float kappa, float rpr, float ca, float cb, float cg, float old_x, float old_t,
                                       float (&new_)[2], float (&dl)[2]) {
  using C = float;
  const C ux_0 = UX(0, 0), ux_p = UX(1, 0);
  const C uy_00 = UY(0, 0), uy_01 = UY(0, 1);
  const C uz_00 = UZ(0, 0), uz_01 = NUZ(0, 0);
  // ux has no unknown at i = 1 (face 1 is the wall): its value there is
  // formed from in-bounds shared-memory neighbours and discarded, so the
  // whole cell stays one branch-free block the scheduler can interleave
  {
    const C ux_m = UX(-1, 0);
    const C ux_jm = UX(0, -1), ux_jp = UX(0, 1);
    const C ux_km = MUX(0), ux_kp = NUX(0);
    const C uy_m0 = UY(-1, 0), uy_m1 = UY(-1, 1);
    const C uz_m0 = UZ(-1, 0), uz_m1 = NUZ(-1, 0);
    C e, gi;
    // advection (ux.c:92-186): invj (l q_m + c q_0 + u q_p) with c = -l - u,
    // l = -0.5 (a q_m' + a' q_0'), u = 0.5 (...), as differences from q_0
    e = (q.xa1 * ux_m + q.xa2 * ux_0) * (ux_m - ux_0) - (q.xa2 * ux_0 + q.xa3 * ux_p) * (ux_p - ux_0);
    e += (q.yb1 * uy_m0 + q.yb2 * uy_00) * (ux_jm - ux_0) - (q.yb1 * uy_m1 + q.yb2 * uy_01) * (ux_jp - ux_0);
    e += (q.zc1 * uz_m0 + q.zc2 * uz_00) * (ux_km - ux_0) - (q.zc1 * uz_m1 + q.zc2 * uz_01) * (ux_kp - ux_0);
    // centrifugal term (:194-226): invj hd (uy averaged to the face)^2
    const C sm = uy_m0 + uy_m1, sp = uy_00 + uy_01;
    e += q.h1 * sm * sm + q.h2 * sp * sp;
    // cross diffusion (:266-375): diffusion_y1 and the uy part of diffusion_a
    // as differences of uy across j, the ux part of diffusion_a, diffusion_z1
    e += q.cy1 * (uy_m1 - uy_m0) + q.cy2 * (uy_01 - uy_00) + q.ca1 * (ux_m + ux_0) +
         q.ca2 * (ux_0 + ux_p) + q.cz1 * ((uz_01 - uz_m1) - (uz_00 - uz_m0));   // coefficients carry nu
    // pressure gradient (:377-394)
    gi = -q.px * (C)(PP(0, 0) - PP(-1, 0));
    ROUTE(im.x, q.lxl * (ux_m - ux_0) + q.lxu * (ux_p - ux_0));        // carries 2 nu
    ROUTE(im.y, q.ly * ((ux_jm - ux_0) + (ux_jp - ux_0)));             // carries nu
    ROUTE(im.z, nu * (lz.l * ux_km + lz.c * ux_0 + lz.u * ux_kp));
    new_[0] = e;
    dl[0] = ca * e + cb * old_x + cg * gi;
  }
  {
    const C t_0 = TT(0, 0);
    const C tim = TT(-1, 0), tip = TT(1, 0), tjm = TT(0, -1), tjp = TT(0, 1);
    const C tkm = MTT(), tkp = NTT(0);
    C e, gi = 0;
    // advection (t.c:88-116) with face velocities ux_0, ux_p, uy_00, uy_01, uz_00, uz_01
    e = q.tx0 * ux_0 * (tim - t_0) - q.tx1 * ux_p * (tip - t_0);
    e += q.ty * uy_00 * (tjm - t_0) - q.ty * uy_01 * (tjp - t_0);
    e += q.tz * uz_00 * (tkm - t_0) - q.tz * uz_01 * (tkp - t_0);
    ROUTE(im.x, rpr * (q.clxl * (tim - t_0) + q.clxu * (tip - t_0)));   // nu kappa/nu
    ROUTE(im.y, rpr * (q.cly * ((tjm - t_0) + (tjp - t_0))));
    ROUTE(im.z, kappa * (lz.l * tkm + lz.c * t_0 + lz.u * tkp));
    new_[1] = e;
    dl[1] = ca * e + cb * old_t + cg * gi;
  }
}


// uy (uy.c) and uz (uz.c) at centre i of line JL
template <class L, int JL, bool TILE, class D>
__device__ __forceinline__ void cell32(const CoefB32 & q, const View<L, float, TILE> & M, const View<L, float, TILE> & V,
                                       const View<L, float, TILE> & N, const D & im, const CoefZ32 & lz, float nu, float,
                                       float, float ca, float cb, float cg, float old_y, float old_z, float (&new_)[2],
                                       float (&dl)[2]) {
  using C = float;
  const C ux_0 = UX(0, 0), ux_1 = UX(1, 0);
  const C uy_0 = UY(0, 0), uy_jp = UY(0, 1);
  const C uz_0 = UZ(0, 0), uz_kp = NUZ(0, 0);
  const double p_0 = PP(0, 0);   // p is double in both modes
  {  // uy
    const C uy_im = UY(-1, 0), uy_ip = UY(1, 0), uy_jm = UY(0, -1);
    const C uy_km = MUY(0), uy_kp = NUY(0);
    const C ux_0m = UX(0, -1), ux_1m = UX(1, -1);
    const C uz_jm = UZ(0, -1), uz_jmkp = NUZ(0, -1);
    C e, gi;
    // advection (uy.c:93-180), as differences from uy_0
    e = q.a1 * (ux_0m + ux_0) * (uy_im - uy_0) - q.a2 * (ux_1m + ux_1) * (uy_ip - uy_0);
    e += q.b * (uy_jm + uy_0) * (uy_jm - uy_0) - q.b * (uy_0 + uy_jp) * (uy_jp - uy_0);
    e += q.c * (uz_jm + uz_0) * (uy_km - uy_0) - q.c * (uz_jmkp + uz_kp) * (uy_kp - uy_0);
    // advection_1 (:188-223): -invjc hd (uy ux averaged to j -/+ 1/2)
    // with the product of the face between the pair's lines, which both use, rounded
    {
      const C lo = uy_jm + uy_0, hi = uy_0 + uy_jp, wlo = ux_0m + ux_1m, whi = ux_0 + ux_1;
      e -= q.h * (JL == 0 ? fmaf(lo, wlo, __fmul_rn(hi, whi)) : fmaf(hi, whi, __fmul_rn(lo, wlo)));
    }
    // diffusion_x1 + diffusion_a (lyx at faces i, i+1 and lxy), diffusion_y1
    // (lyy1 at j-1, j), diffusion_z1 (lyz at k, k+1)
    e += q.p1 * (ux_0 - ux_0m) + q.p2 * (ux_1 - ux_1m) + q.qm * uy_im + q.q0 * uy_0 + q.qp * uy_ip +
         q.yk * ((ux_0 + ux_1) - (ux_0m + ux_1m)) + q.yz * ((uz_kp - uz_jmkp) - (uz_0 - uz_jm));   // carry nu
    gi = -q.py * (C)(p_0 - PP(0, -1));
    ROUTE(im.x, q.lxl * (uy_im - uy_0) + q.lxu * (uy_ip - uy_0));      // carry nu
    ROUTE(im.y, C(2) * (q.ly * ((uy_jm - uy_0) + (uy_jp - uy_0))));
    ROUTE(im.z, nu * (lz.l * uy_km + lz.c * uy_0 + lz.u * uy_kp));
    new_[0] = e;
    dl[0] = ca * e + cb * old_y + cg * gi;
  }
  {  // uz
    const C uz_im = UZ(-1, 0), uz_ip = UZ(1, 0), uz_jm = UZ(0, -1), uz_jp = UZ(0, 1);
    const C uz_km = MUZ();
    const C uy_km = MUY(0), uy_jpkm = MUY(1);
    const C ux_0k = MUX(0), ux_1k = MUX(1);
    C e, gi;
    // advection (uz.c:88-180), as differences from uz_0
    e = q.a1 * (ux_0k + ux_0) * (uz_im - uz_0) - q.a2 * (ux_1k + ux_1) * (uz_ip - uz_0);
    e += q.b * (uy_km + uy_0) * (uz_jm - uz_0) - q.b * (uy_jpkm + uy_jp) * (uz_jp - uz_0);
    e += q.c * (uz_km + uz_0) * (uz_km - uz_0) - q.c * (uz_0 + uz_kp) * (uz_kp - uz_0);
    // diffusion_x1 (lzx at faces i, i+1), diffusion_y1 (lzy at j, j+1)
    e += q.zx1 * (ux_1 - ux_1k) - q.zx0 * (ux_0 - ux_0k) + q.zy * ((uy_jp - uy_jpkm) - (uy_0 - uy_km));   // carry nu
    gi = -lz.ihz * (C)(p_0 - MPP());
    ROUTE(im.x, q.lxl * (uz_im - uz_0) + q.lxu * (uz_ip - uz_0));
    ROUTE(im.y, q.ly * ((uz_jm - uz_0) + (uz_jp - uz_0)));
    ROUTE(im.z, C(2) * nu * (lz.l * uz_km + lz.c * uz_0 + lz.u * uz_kp));
    new_[1] = e;
    dl[1] = ca * e + cb * old_z + cg * gi;
  }
}
#undef ROW_
#undef UX
#undef UY
#undef UZ
#undef TT
#undef PP
#undef NUX
#undef NUY
#undef NUZ
#undef NTT
#undef MUX
#undef MUY
#undef MUZ
#undef MTT
#undef MPP
#undef ROUTE

// One group's state in a thread (as the double one: tc_march.cuh).
template <class L, int GRP, int IMPL, bool TILE>
struct Group<L, GRP, IMPL, float, TILE> {
  using T = float;
  static constexpr int VA = GRP == 0 ? VUX : VUY, VB = GRP == 0 ? VT : VUZ;
  typename std::conditional<GRP == 0, CoefA32, CoefB32>::type q;
  float * na, * nb;          // new source terms of the pair's first line, next plane
  const float * ga, * gb;    // tiles: old source terms (read from global memory)
  const float * oa, * ob;    // old source terms in shared memory
  double * st;
  int ls, pa, pb;
  bool act, acta;

  __device__ __forceinline__ void begin(const Args<float> & A, const Box & x, double * stage, const float * olds, int pr,
                                        int is) {
    const int nx = A.g.nx, ny = A.g.ny, i = x.ib + is;
    act = i <= nx && 2 * pr < x.nl;
    acta = act && (GRP == 1 || i >= 2);   // ux has no unknown at i = 1
    load_coefs32(q, A.cf, i <= nx ? i : 1, A.nu);
    ls = spitch32(nx);
    const int ia = GRP == 0 ? i - 2 : i - 1;
    const size_t qa = pidx(ls, ny, ia, x.j0 + 2 * pr, x.k0), qb = pidx(ls, ny, i - 1, x.j0 + 2 * pr, x.k0);
    na = A.ss.new_[VA] + qa;
    nb = A.ss.new_[VB] + qb;
    ga = TILE && A.rkstep != 0 ? A.ss.old_[VA] + qa : nullptr;
    gb = TILE && A.rkstep != 0 ? A.ss.old_[VB] + qb : nullptr;
    // at i = 1 the old ux term read is the word before the line (discarded)
    oa = olds + (size_t)VA * L::JT * L::OL + 2 * pr * ls + ia;
    ob = olds + (size_t)VB * L::JT * L::OL + 2 * pr * ls + i - 1;
    st = stage + (size_t)(2 * pr * 4) * L::SL;
    // staging positions: unknown 0 of ux is face 2; tiles, which are not solved here, count from face ib + 1
    pa = spad<L::E>(GRP == 0 && !TILE ? is - 2 : is - 1);
    pb = spad<L::E>(is - 1);
  }
  template <class... X>
  __device__ __forceinline__ void below(X &&...) {}
  __device__ __forceinline__ void plane(const Args<float> & A, const CoefZ<float> &, const View<L, float, TILE> & M,
                                        const View<L, float, TILE> & V, const View<L, float, TILE> & N,
                                        const Dirs<IMPL> & im, const Bars<L> & bars, volatile int * abort_flag, int step,
                                        float ca, float cb, float cg) {
    const size_t sp = (size_t)ls * A.g.ny;   // plane stride
    float o_a[2] = {0, 0}, o_b[2] = {0, 0};
    if (A.rkstep != 0) {
      if constexpr (TILE) {
#pragma unroll
        for (int l = 0; l < 2; l++) {
          if (acta) o_a[l] = ga[(size_t)l * ls + step * sp];
          if (act) o_b[l] = gb[(size_t)l * ls + step * sp];
        }
      } else {
        const int buf = (step & 1) * 4 * L::JT * L::OL;
        await(bars.olds(step & 1), (unsigned)(step >> 1) & 1u, abort_flag);
#pragma unroll
        for (int l = 0; l < 2; l++) {
          o_a[l] = oa[buf + l * ls];
          o_b[l] = ob[buf + l * ls];
        }
      }
    }
    const CoefZ32 lz{(float)A.cf.lz_l, (float)A.cf.lz_c, (float)A.cf.lz_u, (float)A.cf.inv_hz};
    const float nu = (float)A.nu, kappa = (float)A.kappa;
    const float rpr = (float)(A.kappa / A.nu);   // the scalar's Laplacians use the centred tables with kappa
    double * sd = st + (size_t)(step & 1) * L::JT * 4 * L::SL;
    auto line = [&](auto jl) {
      constexpr int JL = decltype(jl)::value;
      float e[2], dl[2];
      cell32<L, JL, TILE>(q, M, V, N, im, lz, nu, kappa, rpr, ca, cb, cg, o_a[JL], o_b[JL], e, dl);
      if (acta) {
        na[JL * ls] = e[0];
        sd[(JL * 4 + VA) * L::SL + pa] = (double)dl[0];
      }
      if (act) {
        nb[JL * ls] = e[1];
        sd[(JL * 4 + VB) * L::SL + pb] = (double)dl[1];
      }
    };
    line(std::integral_constant<int, 0>());
    line(std::integral_constant<int, 1>());
    na += sp;
    nb += sp;
  }
};

}  // namespace march
}  // namespace tcgpu
