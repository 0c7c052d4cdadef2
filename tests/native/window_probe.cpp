// Host build of the tile windows (host_common.h) for test_window_limits.py.
#include <cuda_runtime.h>
#define SARBP_HOST_ESTIMATES
static inline float sqrt_estimate(float x) { return x; }
static inline float rcp_estimate(float x) { return x; }
static inline double rsqrt_estimate(double x) { return x; }
static inline int __shfl_sync(unsigned, int v, int) { return v; }
static inline unsigned atomicOr(unsigned *p, unsigned v) { return *p |= v; }
static inline size_t __cvta_generic_to_shared(const void *p) { return reinterpret_cast<size_t>(p); }
static inline int __double2hiint(double) { return 0; }
static inline int __double2loint(double) { return 0; }
static inline double __hiloint2double(int, int) { return 0.0; }
static struct { unsigned x; } threadIdx;
#include "../../uncc_sar_focusing_b200/csrc/host_common.h"

extern "C" int window_probe(double lambda, double dx, double dy, int mx, int *W, int *wsize) {
    double hd;
    sarbp::host::tile_window(lambda, dx, dy, mx, W, wsize, &hd);
    return 0;
}
