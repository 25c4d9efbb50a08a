// Implicit solves of whole lines by warps, with the update of the fields in the last
// direction's store:
//   xsolve_kernel        radial lines longer than the marching kernel's CTAs
//   shared_lines_kernel  periodic (Sherman-Morrison, src/tdm.c:66-106) y and z lines
//                        that share their factors, FP64 contexts
#include <algorithm>

#include "tc_common.cuh"
#include "tc_kernels.h"

namespace tcgpu {

// ------------------------------------------------------------ solves from shared memory
// LN lines of up to 32 E unknowns by one warp, lane t owning elements tE .. tE + E - 1
// (at(l, m): element tE + m of line l; keep(m): whether it takes its solution). The
// recurrences, their order of operations and the scan products are those of
// march::solve_lines; the factors are read from shared memory as they are used (rows
// f, g, w of 32 E, element tE + m at 32 m + t, then the scan products up and down),
// which costs a conflict-free load for LN multiply-adds and no registers.
// SINGLE: FP32-storage rows, pivots taken into the right-hand side first.
template <int E, int LN, bool SINGLE, class At, class Keep>
__device__ __forceinline__ void line_solve(const double * tab, int lane, At at, Keep keep) {
  const double * const f = tab + lane, * const g = f + 32 * E, * const w = g + 32 * E, * const sc = w + 32 * E;
  double r[LN][E], B[LN], p[LN];
#pragma unroll
  for (int m = 0; m < E; m++) {
    const double s = SINGLE ? w[m * 32] : 1.;
#pragma unroll
    for (int l = 0; l < LN; l++) r[l][m] = SINGLE ? __dmul_rn(s, at(l, m)) : at(l, m);
  }
#pragma unroll
  for (int l = 0; l < LN; l++) B[l] = r[l][0];
#pragma unroll
  for (int m = 1; m < E; m++) {
    const double c = f[m * 32];
#pragma unroll
    for (int l = 0; l < LN; l++) B[l] = fma(c, B[l], r[l][m]);
  }
#pragma unroll
  for (int q = 0; q < 5; q++) {
    const double c = sc[q * 32];
#pragma unroll
    for (int l = 0; l < LN; l++) B[l] = fma(c, __shfl_up_sync(0xffffffffu, B[l], 1 << q), B[l]);
  }
#pragma unroll
  for (int l = 0; l < LN; l++) p[l] = __shfl_up_sync(0xffffffffu, B[l], 1);   // lane 0: f[0] = 0
#pragma unroll
  for (int m = 0; m < E; m++) {
    const double c = f[m * 32];
#pragma unroll
    for (int l = 0; l < LN; l++) p[l] = r[l][m] = fma(c, p[l], r[l][m]);
  }
#pragma unroll
  for (int l = 0; l < LN; l++) B[l] = r[l][E - 1];
#pragma unroll
  for (int m = E - 2; m >= 0; m--) {
    const double c = g[m * 32];
#pragma unroll
    for (int l = 0; l < LN; l++) B[l] = fma(c, B[l], r[l][m]);
  }
#pragma unroll
  for (int q = 0; q < 5; q++) {
    const double c = sc[(5 + q) * 32];
#pragma unroll
    for (int l = 0; l < LN; l++) B[l] = fma(c, __shfl_down_sync(0xffffffffu, B[l], 1 << q), B[l]);
  }
#pragma unroll
  for (int l = 0; l < LN; l++) p[l] = __shfl_down_sync(0xffffffffu, B[l], 1);   // lane 31: g of the last is 0
#pragma unroll
  for (int m = E - 1; m >= 0; m--) {
    const double c = g[m * 32], s = SINGLE ? 1. : w[m * 32];
#pragma unroll
    for (int l = 0; l < LN; l++) {
      p[l] = fma(c, p[l], r[l][m]);
      if (keep(m)) at(l, m) = SINGLE ? p[l] : s * p[l];
    }
  }
}

// ------------------------------------------------------------ radial lines
// Radial implicit solves of lines longer than one CTA's field threads (the marching
// kernel's tile mode leaves its increments unsolved), and, where no other direction
// is implicit, the update u + delta with walls and images in the store.
// One CTA per SM with one variable's factors in shared memory; each warp walks over
// pairs of lines, the next pair's increments and fields under way (cp.async) while it
// solves and stores the present one.
// Bound: HBM, 16 bytes a value (24 with the update). One line per warp with the
// factors loaded for each: solve and update 2.07 ms a step at 384 x 256 x 128, 0.85
// here (floor 0.58).
__host__ __device__ constexpr int xsolve_warps(int E) { return E <= 12 ? 8 : E <= 16 ? 6 : E <= 24 ? 4 : 3; }
template <class T>
__device__ __forceinline__ void cp_async(T * dst, const T * src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], %2;" ::"r"(smem_u32(dst)), "l"(src), "n"(sizeof(T)) : "memory");
}
template <int E, class T>
struct XStage {   // a pair of lines
  double x[2][32 * E + 32];   // increments, then solutions; element e at e + e / E
  T u[2][32 * E];
};
template <int E, class T>
__global__ void __launch_bounds__(32 * xsolve_warps(E)) xsolve_kernel(Geo g, Bc bc, XFactors xf, int rk, DeltaSet ds,
                                                                      FieldsT<T> in, FieldsT<T> out, bool update) {
  constexpr bool SINGLE = sizeof(T) == 4;
  constexpr int NW = xsolve_warps(E), ROWS = 3 * 32 * E + 10 * 32;
  extern __shared__ double xs_tab[];
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, v = blockIdx.y;
  XStage<E, T> * const stage = reinterpret_cast<XStage<E, T> *>(xs_tab + ROWS) + 2 * wid;
  const int n = v == VUX ? xf.n[VUX] : xf.n[VUY], ny = g.ny, nz = g.nz, lines = ny * nz;
  double * const d = v == VUX ? ds.d[0] : v == VUY ? ds.d[1] : v == VUZ ? ds.d[2] : ds.d[3];   // line (j, k): n values
  const T * const src = v == VUX ? in.ux : v == VUY ? in.uy : v == VUZ ? in.uz : in.t;
  T * const dst = v == VUX ? out.ux : v == VUY ? out.uy : v == VUZ ? out.uz : out.t;
  // element of unknown 0 in a row, and the elements of the walls
  const int o = v == VUX ? (int)sidx_f<T>(g, 2, 0, 0) : 1, om = o - 1, op = o + n;
  const int len = v == VUX ? srow_f<T>(g) : srow_c<T>(g);
  const T wm = (T)(v == VUY ? bc.uy_xm : v == VT ? bc.t_xm : 0.), wp = (T)(v == VUY ? bc.uy_xp : v == VT ? bc.t_xp : 0.);
  auto at = [&](int jj, int kk) { return (size_t)len * ((size_t)jj + (size_t)(ny + 2) * kk); };
  auto load = [&](int line0, XStage<E, T> & st) {   // lines past the last leave their slots as they are
#pragma unroll
    for (int l = 0; l < 2; l++) {
      const int line = line0 + l;
      if (line < lines) {
        const double * const dl = d + (size_t)line * n;
        const T * const ul = src + at(line % ny + 1, line / ny + 1) + o;
#pragma unroll
        for (int m = 0; m < E; m++) {
          const int e = m * 32 + lane;
          if (e < n) {
            cp_async(&st.x[l][e + e / E], dl + e);
            if (update) cp_async(&st.u[l][e], ul + e);
          }
        }
      }
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  // rows past n stay zero in every slot
  for (int q = 0; q < 2; q++)
    for (int l = 0; l < 2; l++)
      for (int e = n + lane; e < 32 * E; e += 32) stage[q].x[l][e + e / E] = 0.;
  const int step = 2 * NW * gridDim.x;
  int line0 = 2 * (blockIdx.x * NW + wid), buf = 0;
  load(line0, stage[0]);
  {
    const size_t fo = (size_t)(rk * 4 + v) * xf.stride;
    for (int e = threadIdx.x; e < 32 * E; e += 32 * NW) {
      const double f = xf.f[fo + e], gg = xf.g[fo + e], w = xf.w[fo + e];
      xs_tab[e] = SINGLE ? __dmul_rn(-w, f) : f;
      xs_tab[32 * E + e] = SINGLE ? -gg : gg;
      xs_tab[2 * 32 * E + e] = w;
    }
    for (int e = threadIdx.x; e < 10 * 32; e += 32 * NW)
      xs_tab[3 * 32 * E + e] = xf.scan[(size_t)(rk * 4 + v) * XSCAN_ROWS * 32 + e];
  }
  __syncthreads();
  for (; line0 < lines; line0 += step, buf ^= 1) {
    load(line0 + step, stage[buf ^ 1]);
    asm volatile("cp.async.wait_group 1;" ::: "memory");
    __syncwarp();
    XStage<E, T> & st = stage[buf];
    line_solve<E, 2, SINGLE>(xs_tab, lane, [&](int l, int m) -> double & { return st.x[l][lane * (E + 1) + m]; },
                             [&](int m) { return lane * E + m < n; });
    __syncwarp();
#pragma unroll
    for (int l = 0; l < 2; l++) {
      const int line = line0 + l;
      if (line >= lines) break;
      const double * const x = st.x[l];
      if (!update) {
#pragma unroll
        for (int m = 0; m < E; m++) {
          const int e = m * 32 + lane;
          if (e < n) d[(size_t)line * n + e] = x[e + e / E];
        }
        continue;
      }
      const int j = line % ny + 1, k = line / ny + 1;
      auto put = [&](int jj, int kk) {
        T * const row = dst + at(jj, kk);
#pragma unroll
        for (int m = 0; m < E; m++) {
          const int e = m * 32 + lane;
          if (e < n) row[o + e] = (T)((double)st.u[l][e] + x[e + e / E]);
        }
        if (lane == 0) row[om] = wm;
        if (lane == 1) row[op] = wp;
      };
      put(j, k);
      if (j == 1 || j == ny || k == 1 || k == nz) for_images(j, k, ny, nz, put);
    }
    __syncwarp();   // the slot is filled again in the next turn
  }
}

// elements per lane of these lines (XFactors::ne): predict_warps, predict_warps32
#define X_LINES(X) X(12, double) X(16, double) X(24, double) X(32, double) X(16, float) X(32, float)
template <int E, class T>
constexpr size_t xsolve_smem() { return sizeof(double) * (3 * 32 * E + 320) + 2 * xsolve_warps(E) * sizeof(XStage<E, T>); }

void launch_xsolve(const Geo & g, const Bc & bc, const XFactors & xf, int rkstep, const DeltaSet & ds,
                   const FieldBufs & in, const FieldBufs & out, bool update, cudaStream_t st) {
  int dev = 0, sms = 0;
  if (cudaGetDevice(&dev) != cudaSuccess ||
      cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess) {
    sms = 148;
    cudaGetLastError();
  }
  const int pairs = (g.ny * g.nz + 1) / 2, per = sms > 4 ? sms / 4 : 1;
  switch (xf.ne + (xf.single ? 64 : 0)) {
#define X(EE, T)                                                                                             \
  case EE + (sizeof(T) == 4 ? 64 : 0): {                                                                     \
    constexpr int NW = xsolve_warps(EE);                                                                     \
    const dim3 grid(std::min(per, (pairs + NW - 1) / NW), 4);                                                \
    xsolve_kernel<EE, T><<<grid, 32 * NW, xsolve_smem<EE, T>(), st>>>(g, bc, xf, rkstep, ds, in.as<T>(),     \
                                                                      out.as<T>(), update);                  \
    break;                                                                                                   \
  }
    X_LINES(X)
#undef X
  }
}

// ------------------------------------------------------------ periodic lines, shared factors
// Periodic y and z solves where all lines of a variable share their factors (z
// always; y on planar grids), FP64 contexts, lines of up to 1024 points: one launch
// for the four variables, and in the last implicit direction the update u + delta
// (walls, images) in the store, so that the increments are not written and read again.
// A CTA takes 16 radial indices; thread (t, c) keeps the E values of chunk c of line t
// in registers from the load to the store (half warps read and write whole rows of
// 16), so that shared memory holds only the factors, read as broadcasts, and the
// chunks' boundary values: each thread walks those before (after) its own with the
// chunks' tabulated products. The Sherman-Morrison correction needs three values a line.
// Bound: HBM, 16 bytes a value (24 with the update). Solves and update of a step of
// 192 x 512 x 256: 4.68 ms with a launch a variable and the update apart, 3.68 with
// the lines staged in shared memory and solved by warps, 2.96 here (floor 1.9).
struct LineTable {   // doubles of one (substep, variable): f, g, w, q1 in order, chunk products, then l, u, 1 / den
  static __host__ __device__ constexpr int rows(int E, int C) { return 4 * E * C; }
  static __host__ __device__ constexpr int size(int E, int C) { return 4 * E * C + 2 * C + 4; }
};
// values per thread and chunks of lines of n points (an even number of chunks: whole warps)
static int line_values(int n) { return n <= 64 ? 4 : n <= 256 ? 8 : n <= 512 ? 16 : n <= 1024 ? 32 : 0; }
static int line_chunks(int n, int E) { return ((n + E - 1) / E + 1) & ~1; }
struct LineArgs {
  Geo g;
  Bc bc;
  DeltaSet ds;
  FieldsT<double> in, out;
  const double * table;    // [4][LineTable::size(E, C)]
  int n, C;                // points and chunks per line
  bool z;                  // lines along z (else y)
};
constexpr int LINE_PT = 16;
template <int E, bool UPDATE>
__global__ void __launch_bounds__(512, E <= 16 ? 2 : 1) shared_lines_kernel(LineArgs A) {
  constexpr bool EARLY = UPDATE && E <= 8;   // the fields' values beside the increments, where registers hold both
  constexpr int PT = LINE_PT;
  extern __shared__ __align__(16) double tab[];
  const int v = blockIdx.z, n = A.n, C = A.C, nx = A.g.nx, ny = A.g.ny, nz = A.g.nz;
  const int n_i = v == VUX ? nx - 1 : nx, ii0 = blockIdx.x * PT;
  if (ii0 >= n_i) return;
  const int o = blockIdx.y;   // k - 1 of y lines, j - 1 of z lines
  const int t = threadIdx.x % PT, c = threadIdx.x / PT, j0 = c * E;
  const bool mine = ii0 + t < n_i;
  double * const base = A.ds.d[v] + ii0 + t + (A.z ? (size_t)n_i * o : (size_t)n_i * ny * o);
  const size_t es = A.z ? (size_t)n_i * ny : (size_t)n_i;
  const int size = LineTable::size(E, C);
  const double * const src = A.table + (size_t)v * size;
  for (int q = 2 * threadIdx.x; q < size; q += 2 * blockDim.x)
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_u32(tab + q)), "l"(src + q) : "memory");
  double r[E];
#pragma unroll
  for (int m = 0; m < E; m++) r[m] = mine && j0 + m < n ? base[(size_t)(j0 + m) * es] : 0.;
  // unknown ii of a line is element ii + 1 of its row (ux: face ii + 2, element ii + 1)
  const int len = v == VUX ? nx + 1 : nx + 2, e = ii0 + t + 1;
  const double * const in = (v == VUX ? A.in.ux : v == VUY ? A.in.uy : v == VUZ ? A.in.uz : A.in.t) + e;
  auto at = [&](int jj, int kk) { return (size_t)len * ((size_t)jj + (size_t)(ny + 2) * kk); };
  const size_t a0 = A.z ? at(o + 1, j0 + 1) : at(j0 + 1, o + 1), as = A.z ? (size_t)len * (ny + 2) : (size_t)len;
  double u[EARLY ? E : 1];
  if (EARLY) {
#pragma unroll
    for (int m = 0; m < E; m++) u[m] = mine && j0 + m < n ? in[a0 + m * as] : 0.;
  }
  const int NP = E * C;
  const double * const f = tab + j0, * const g = f + NP, * const w = g + NP, * const q1 = w + NP;
  const double * const prod = tab + 4 * NP, * const k = prod + 2 * C;
  double * const bf = tab + size, * const bb = bf + C * PT, * const edge = bb + C * PT;
  asm volatile("cp.async.wait_all;" ::: "memory");
  __syncthreads();
  // factors in pairs: half the shared-memory reads
  auto two = [](const double * q) { return *reinterpret_cast<const double2 *>(q); };
  double p = 0.;
#pragma unroll
  for (int m = 0; m < E; m += 2) {
    const double2 a = two(f + m);
    p = m == 0 ? r[0] : fma(a.x, p, r[m]);
    p = fma(a.y, p, r[m + 1]);
  }
  bf[threadIdx.x] = p;
  __syncthreads();
  p = 0.;
#pragma unroll 8
  for (int q = 0; q < c; q++) p = fma(prod[q], p, bf[q * PT + t]);
#pragma unroll
  for (int m = 0; m < E; m += 2) {
    const double2 a = two(f + m);
    r[m] = fma(a.x, p, r[m]);
    p = r[m + 1] = fma(a.y, r[m], r[m + 1]);
  }
  if (c == (n - 1) / E) {   // the last row keeps its right-hand side (f = 0)
#pragma unroll
    for (int m = 0; m < E; m++)
      if (j0 + m == n - 1) edge[t] = r[m];
  }
#pragma unroll
  for (int m = E - 2; m >= 0; m -= 2) {
    const double2 a = two(g + m);
    p = m == E - 2 ? p : fma(a.y, p, r[m + 1]);
    p = fma(a.x, p, r[m]);
  }
  bb[threadIdx.x] = p;
  __syncthreads();
  p = 0.;
#pragma unroll 8
  for (int q = C - 1; q > c; q--) p = fma(prod[C + q], p, bb[q * PT + t]);
#pragma unroll
  for (int m = E - 2; m >= 0; m -= 2) {
    const double2 a = two(g + m), b = two(w + m);
    p = fma(a.y, p, r[m + 1]);
    r[m + 1] = b.y * p;
    p = fma(a.x, p, r[m]);
    r[m] = b.x * p;
  }
  if (c == 0) edge[PT + t] = r[0];
  if (c == (n - 2) / E) {
#pragma unroll
    for (int m = 0; m < E; m++)
      if (j0 + m == n - 2) edge[2 * PT + t] = r[m];
  }
  __syncthreads();
  // the last unknown (src/tdm.c:88-96); q1 is 1 and w 0 in its row
  const double last = (edge[t] - k[1] * edge[PT + t] - k[0] * edge[2 * PT + t]) * k[2];
  if (!mine) return;
#pragma unroll
  for (int m = 0; m < E; m += 2) {
    const double2 a = two(q1 + m);
    r[m] = fma(last, a.x, r[m]);
    r[m + 1] = fma(last, a.y, r[m + 1]);
  }
  if (!UPDATE) {
#pragma unroll
    for (int m = 0; m < E; m++)
      if (j0 + m < n) base[(size_t)(j0 + m) * es] = r[m];
    return;
  }
  if (EARLY) {
#pragma unroll
    for (int m = 0; m < E; m++) r[m] += u[m];
  } else {
#pragma unroll
    for (int m = 0; m < E; m++)
      if (j0 + m < n) r[m] += in[a0 + m * as];
  }
  double * const out = (v == VUX ? A.out.ux : v == VUY ? A.out.uy : v == VUZ ? A.out.uz : A.out.t) + e;
  const double wm = v == VUY ? A.bc.uy_xm : v == VT ? A.bc.t_xm : 0., wp = v == VUY ? A.bc.uy_xp : v == VT ? A.bc.t_xp : 0.;
  const bool first = e == 1, lst = e == n_i, oedge = o == 0 || o == (A.z ? ny : nz) - 1;
#pragma unroll
  for (int m = 0; m < E; m++) {
    const int q = j0 + m;
    if (q >= n) break;
    auto put = [&](size_t a) {
      out[a] = r[m];
      if (first) out[a - 1] = wm;
      if (lst) out[a + 1] = wp;
    };
    put(a0 + m * as);
    if (oedge || q == 0 || q == n - 1)
      for_images(A.z ? o + 1 : q + 1, A.z ? q + 1 : o + 1, ny, nz, [&](int jj, int kk) { put(at(jj, kk)); });
  }
}

// at most 42 KB
static size_t shared_lines_smem(int E, int C) { return sizeof(double) * (LineTable::size(E, C) + (2 * C + 3) * LINE_PT); }

size_t shared_lines_table(int n) {
  const int E = line_values(n);
  return E ? (size_t)12 * LineTable::size(E, line_chunks(n, E)) : 0;
}

void allow_lines_smem() {
#define X(EE, T) \
  cudaFuncSetAttribute(xsolve_kernel<EE, T>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)xsolve_smem<EE, T>());
  X_LINES(X)
#undef X
}

// all four variables along one direction; table: shared_lines_table(n) doubles
void launch_shared_lines(const Geo & g, const Bc & bc, const DeltaSet & ds, const FieldBufs & in, const FieldBufs & out,
                         const double * table, int rkstep, bool z, bool update, cudaStream_t st) {
  LineArgs A{g, bc, ds, in.as<double>(), out.as<double>(), table, z ? g.nz : g.ny, 0, z};
  const int E = line_values(A.n);
  A.C = line_chunks(A.n, E);
  A.table += (size_t)rkstep * 4 * LineTable::size(E, A.C);
  const dim3 grid((g.nx + LINE_PT - 1) / LINE_PT, z ? g.ny : g.nz, 4);
  const unsigned threads = LINE_PT * A.C;
  const size_t smem = shared_lines_smem(E, A.C);
#define X(EE)                                                                          \
  if (E == EE && update) shared_lines_kernel<EE, true><<<grid, threads, smem, st>>>(A); \
  else if (E == EE) shared_lines_kernel<EE, false><<<grid, threads, smem, st>>>(A);
  X(4) X(8) X(16) X(32)
#undef X
}

// The tables of both directions: one block per (direction, substep, variable). As
// in xfactor_kernel the pivots are ratios of minors (of the reduced system of n - 1
// rows): with the pivots 1 / w, f_e = -l w_{e-1} and g_e = -u w_{e+1}. q1 solves the
// reduced system for the right-hand side (-l, 0, ..., 0, -u). Doubled prefactors:
// uy-y and t-y (uy.c:541, t.c:348), uz-z (uz.c:451).
constexpr int SHARED_LINE_MAX = 1024;
__global__ void __launch_bounds__(256) shared_factor_kernel(YZFactors yf, int ny, int nz, int ey, int ez, int cy, int cz,
                                                            const double * __restrict__ dtp, double nu, double kappa) {
  __shared__ double sw[SHARED_LINE_MAX], st[SHARED_LINE_MAX];
  const bool z = blockIdx.x >= 12;
  if ((z ? yf.tz : yf.ty) == nullptr) return;
  const int rv = blockIdx.x % 12, rk = rv / 4, var = rv % 4, tid = threadIdx.x;
  const int n = z ? nz : ny, E = z ? ez : ey, C = z ? cz : cy, N = E * C, m = n - 1;
  double * const tab = (z ? yf.tz : yf.ty) + (size_t)rv * LineTable::size(E, C);
  double pf = 0.5 * rk_gamma(rk) * (*dtp) * (var == VT ? kappa : nu);
  if (z ? var == VUZ : (var == VUY || var == VT)) pf = 2. * pf;
  const double l = -pf * (z ? yf.lapz_l : yf.lapy_l[var][0]), c = 1. - pf * (z ? yf.lapz_c : yf.lapy_c[var][0]);
  const double u = -pf * (z ? yf.lapz_u : yf.lapy_u[var][0]);
  if (tid == 0) {
    const double lu = l * u;
    double t2 = 0., t1 = 1.;   // minors e - 2 and e - 1, scaled together
    for (int e = 0; e < m; e++) {
      const double t = fma(c, t1, -lu * t2);
      st[e] = t;
      sw[e] = t1;
      t2 = t1;
      t1 = t;
      const double a = fabs(t1);
      if (a > 0x1p256) { t1 *= 0x1p-256; t2 *= 0x1p-256; }
      else if (a < 0x1p-256) { t1 *= 0x1p256; t2 *= 0x1p256; }
    }
  }
  __syncthreads();
  for (int e = tid; e < m; e += blockDim.x) sw[e] = sw[e] / st[e];
  __syncthreads();
  auto fe = [&](int e) { return e > 0 && e < m ? -l * sw[e - 1] : 0.; };
  auto ge = [&](int e) { return e < m - 1 ? -u * sw[e + 1] : 0.; };
  for (int e = tid; e < N; e += blockDim.x) {
    tab[e] = fe(e);
    tab[N + e] = ge(e);
    tab[2 * N + e] = e < m ? sw[e] : 0.;
  }
  if (tid >= 64 && tid < 64 + 2 * C) {   // products over the chunks
    const int q = (tid - 64) % C;
    double a = 1.;
    for (int e = q * E; e < (q + 1) * E; e++) a *= tid - 64 < C ? fe(e) : ge(e);
    tab[4 * N + tid - 64] = a;
  }
  if (tid == 0) {
    double p = -l;
    st[0] = p;
    for (int e = 1; e < m; e++) {
      p = fma(fe(e), p, e == m - 1 ? -u : 0.);
      st[e] = p;
    }
    double x = 0.;
    for (int e = m - 1; e >= 0; e--) {
      x = fma(ge(e), x, st[e]);
      st[e] = x;
    }
    const double den = c + u * (sw[0] * st[0]) + l * (sw[m - 1] * st[m - 1]);
    double * const k = tab + 4 * N + 2 * C;
    k[0] = l;
    k[1] = u;
    k[2] = fabs(den) < 2.220446049250313e-16 ? 0. : 1. / den;
  }
  __syncthreads();
  for (int e = tid; e < N; e += blockDim.x) tab[3 * N + e] = e < m ? sw[e] * st[e] : e == m ? 1. : 0.;
}

void launch_shared_factors(const Geo & g, const YZFactors & yf, const double * dtp, double nu, double kappa,
                           cudaStream_t st) {
  const int ey = line_values(g.ny), ez = line_values(g.nz);
  shared_factor_kernel<<<24, 256, 0, st>>>(yf, g.ny, g.nz, ey, ez, ey ? line_chunks(g.ny, ey) : 0,
                                           ez ? line_chunks(g.nz, ez) : 0, dtp, nu, kappa);
}

}  // namespace tcgpu
