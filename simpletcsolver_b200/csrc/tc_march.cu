// Launchers of the predict stage (tc_march.cuh): the choice of the instance and
// of the planes per CTA, and the self-test of the kernels' bounded waits.
#include "tc_march.cuh"
#include "tc_march_launch.cuh"

namespace tcgpu {

// Planes per CTA of a marching launch of `columns` CTAs per plane chunk: the
// divisor of nz (up to TC_MARCH_KC) with the least waves x (planes +
// TC_MARCH_START), where TC_MARCH_START planes stand for a CTA's start (barriers,
// coefficients, the first planes' copies, the first solve), which nothing overlaps
// at one CTA per SM. Large grids take long chunks, whose two halo planes and
// starts cost little; small ones take short chunks, down to single planes, so that
// every SM has one (64 x 8 x 32: 54 us a launch in the former chunks of 16 planes
// on 8 SMs, 13 in single planes on 32).
#ifndef TC_MARCH_KC
#define TC_MARCH_KC 64
#endif
#ifndef TC_MARCH_START
#define TC_MARCH_START 3
#endif
int march_planes(long long columns, int nz, int per_sm) {
  int dev = 0, sms = 0;
  // a failed query falls back to 148 SMs and clears its own error
  if (cudaGetDevice(&dev) != cudaSuccess ||
      cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess) {
    sms = 0;
    cudaGetLastError();
  }
  const long long slots = (long long)(sms > 0 ? sms : 148) * per_sm;
  int best = 1;
  long long least = -1;
  for (int kc = 1; kc <= nz && kc <= TC_MARCH_KC; kc++) {
    if (nz % kc) continue;
    const long long blocks = columns * (nz / kc), waves = (blocks + slots - 1) / slots;
    const long long cost = waves * (kc + TC_MARCH_START);
    if (least < 0 || cost <= least) {
      least = cost;
      best = kc;
    }
  }
  return best;
}

void launch_predict_march(const Geo & g, const Bc & bc, const Coefs & cf, const XFactors & xf, double nu,
                          double kappa, const FieldBufs & in, const FieldBufs & out, const SrcBufs & ss,
                          const DeltaSet & ds, const double * dtp, int rkstep, int mode, unsigned * status,
                          cudaStream_t st) {
  const int mask = (bc.implicit[0] ? 1 : 0) | (bc.implicit[1] ? 2 : 0) | (bc.implicit[2] ? 4 : 0);
  const bool tiles = g.nx > 256;   // wider than a CTA's field threads: increments only, solved afterwards
  if (in.bytes == 4) {
    march::Args<float> A{g, bc, cf, xf, nu, kappa, in.as<float>(), out.as<float>(), ss.as<float>(), ds, rkstep, mode, 0,
                         status};
    if (tiles) A.mode = PREDICT_DELTA;
    if (mask == 1 && !tiles) march::launch<1, float>(A, tiles, dtp, st);
    else if (mask == 7 && !tiles) march::launch<7, float>(A, tiles, dtp, st);
    else if (mask == 0 && !tiles) march::launch<0, float>(A, tiles, dtp, st);
    else march::launch<-1, float>(A, tiles, dtp, st);
    return;
  }
  using T = double;
  march::Args<T> A{g, bc, cf, xf, nu, kappa, in.as<T>(), out.as<T>(), ss.as<T>(), ds, rkstep, mode, 0, status};
  if (tiles) A.mode = PREDICT_DELTA;
  // the common masks have instances of their own; the others, and tiles, read the
  // directions at run time (which spills: tiles 0.79 ms at 384 x 256 x 128 that
  // way, 0.52 with the mask compiled in)
  if (A.ss.frc[0]) {
    if (mask == 1 && !tiles) march::launch<9, T>(A, tiles, dtp, st);
    else march::launch<-2, T>(A, tiles, dtp, st);
  }
  else if (mask == 1) march::launch<1, T>(A, tiles, dtp, st);
  else if (mask == 7 && !tiles) march::launch<7, T>(A, tiles, dtp, st);
  else if (mask == 0 && !tiles) march::launch<0, T>(A, tiles, dtp, st);
  else march::launch<-1, T>(A, tiles, dtp, st);
}

// Self-test of the bounded waits: an mbarrier expects 16 bytes that no copy
// will ever deliver; every thread's wait must give up after kWaitCycles and the
// kernel report ST_TIMEOUT and return (the same wait the predict kernel uses).
__global__ void wait_selftest_kernel(unsigned * status) {
  __shared__ __align__(8) unsigned long long bar;
  if (threadIdx.x == 0) {
    mbar_init(&bar, 1);
    fence_mbar_init();
  }
  __syncthreads();
  if (threadIdx.x == 0) mbar_expect_tx(&bar, 16);   // the only arrival; its bytes never come
  __syncthreads();
  const bool ok = mbar_wait(&bar, 0);
  if (__syncthreads_or(!ok) && threadIdx.x == 0) atomicOr(status, ST_TIMEOUT);
}

void launch_wait_selftest(unsigned * status, cudaStream_t st) { wait_selftest_kernel<<<1, 64, 0, st>>>(status); }

// Self-test of the predict's way out: every plane announces 16 bytes more than its
// copies bring, so no plane ever arrives, and every CTA must give up, store no field and
// report ST_TIMEOUT. zeros: what the kernel reads, kept: the fields it would write.
void launch_predict_selftest(const PredictSelftest & b, unsigned * status, cudaStream_t st) {
  Geo g{};
  g.nx = PredictSelftest::NX;
  g.ny = PredictSelftest::NY;
  g.nz = PredictSelftest::NZ;
  constexpr size_t F = PredictSelftest::FIELD;
  march::Args<double> A{};
  A.g = g;
  A.cf.tab = b.zeros;
  A.in = FieldsT<double>{b.zeros, b.zeros, b.zeros, b.zeros, b.zeros, b.zeros};
  A.out = FieldsT<double>{b.kept, b.kept + F, b.kept + 2 * F, nullptr, nullptr, b.kept + 3 * F};
  for (int v = 0; v < 4; v++) {
    A.ss.old_[v] = b.zeros;
    A.ss.new_[v] = b.terms;
  }
  A.rkstep = 1;
  A.mode = PREDICT_APPLY;
  A.status = status;
  A.lost = 16;
  march::launch<0, double>(A, false, b.zeros, st);
}

}  // namespace tcgpu
