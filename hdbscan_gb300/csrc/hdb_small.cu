// Launcher of the small-window kernel (hdb_small.cuh).
#include "hdb_launch.h"
#include "hdb_registry.h"
#include "hdb_small.h"
#include "hdb_small.cuh"

namespace hdb {
namespace {

template <typename Real>
cudaError_t launch(const ForwardArgs& f, const SmallArgs& s, int windows, int nmax, cudaStream_t stream, int priority) {
    return launch_ex(hdb_small_kernel<Real>, (unsigned)windows, nmax <= 32 ? 64u : (nmax <= 64 ? 128u : 256u), SmallLayout<Real>::bytes(nmax),
                     stream, priority, 1, f, s);
}

template <typename Real>
cudaError_t prepare(int nmax) {
    return raise_dynamic_smem((const void*)hdb_small_kernel<Real>, SmallLayout<Real>::bytes(nmax));
}

}  // namespace

cudaError_t small_launch(int precision, const ForwardArgs& f, const SmallArgs& s, int windows, int nmax,
                         cudaStream_t stream, int priority) {
    return precision == 0 ? launch<float>(f, s, windows, nmax, stream, priority)
                          : launch<double>(f, s, windows, nmax, stream, priority);
}

cudaError_t small_prepare(int precision, int nmax) { return precision == 0 ? prepare<float>(nmax) : prepare<double>(nmax); }

bool small_window(int precision, int n, int D, bool unit_core, int windows, int sms) {
    // One CTA computes all distances, which bounds n^2 D.  float32, device time of a
    // batch here and in the general form: 128 points x 64 dims 91 and 112 us (one
    // window), 189 and 323 us (600); x 256 dims 247 and 144 us (one).  float64 runs
    // at two operations a clock on an SM, roots included: 32 x 16 dims 86 and 160 us
    // (one), 121 and 289 us (600); 1500 windows of 16 to 200 points (6 dims) took
    // 1.09 ms with those up to 128 points here, 0.85 ms without.
    const double work = (double)n * n * D;
    if (precision != 0) return n <= 32 && work <= 3.2e4;
    if (n > kSmallMax || work > 1.1e6) return false;
    // Above 96 points two CTAs fill an SM's shared memory; past one wave of them
    // the register form, with no cores to compute, is faster (600 windows of
    // 128 x 4: 132 and 99 us).
    return !(n > 96 && unit_core && D <= 16 && windows > 2 * sms);
}

}  // namespace hdb
