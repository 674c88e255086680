// Jacobian determinant on device pointers without any allocation.
//
// Some callers cannot let a library allocate device memory when they need a
// Jacobian map:
// * hosts that fix their device-memory budget at start-up (real-time and
//   embedded systems), where a later cudaMalloc may fail or, because
//   cudaMalloc and cudaFree can synchronise the device, stall a loop that
//   has a deadline;
// * processes whose device memory is already handed out by another
//   allocator (a framework's caching allocator that reserved it), so an
//   allocation of the library's own fails;
// * runtimes without an allocator of their own, which pass the library
//   pointers into memory they manage.
// The kernel behind it takes its geometry as a parameter and uses no device
// memory of its own.  (dtb_jacobian_device does the same today; this entry
// point is the one that promises it, with any layout and order through one
// kernel.)
//
// The volume limit, NOALLOC_MAX_TILES tiles of 32 x 8 x 32 voxels, is part of
// the interface.
#include <cuda_runtime.h>

#include <cstdio>

#include "dt_internal.h"

using namespace dtb;

namespace {

constexpr int NOALLOC_MAX_TILES = 16384;

void report(int line, const char *function, const char *message) {
    disptools_error_state *e = disptools_get_error();
    e->error = true;
    e->line = line;
    std::snprintf(e->file, sizeof e->file, "%s", __FILE__);
    std::snprintf(e->function, sizeof e->function, "%s", function);
    std::snprintf(e->message, sizeof e->message, "%s", message);
    e->trace[0] = '\0';
}

int num_sms() {
    int dev = 0, v = 0;
    if (cudaGetDevice(&dev) != cudaSuccess ||
        cudaDeviceGetAttribute(&v, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess) {
        cudaGetLastError();
        v = 0;
    }
    return v > 0 ? v : 148;
}

template <typename T>
int jacobian_noalloc(size_t nx, size_t ny, size_t nz, double dx, double dy, double dz, int order, const T *field,
                     T *J, cudaStream_t s) {
    const int bz = nz < 32 ? (int) nz : 32;
    const long long tiles = (long long) ((nx + BX - 1) / BX) * (long long) ((ny + BY - 1) / BY) *
                            (long long) ((nz + bz - 1) / bz);
    if (tiles > NOALLOC_MAX_TILES) {
        char m[256];
        std::snprintf(m, sizeof m,
                      "volume too large for dtb_jacobian_device_noalloc: %lld tiles of %dx%dx%d voxels, "
                      "its limit is %d (use dtb_jacobian_device)",
                      tiles, BX, BY, bz, NOALLOC_MAX_TILES);
        report(__LINE__, __func__, m);
        return DTB_ERR_ARGUMENT;
    }
    Geom g = {};
    g.nx = (int) nx;
    g.ny = (int) ny;
    g.nz = (int) nz;
    g.order = order;
    g.ys = (long long) nx;
    g.zs = (long long) nx * ny;
    g.cs = (long long) nx * ny * nz;
    const double sp[3] = {dx, dy, dz};
    for (int a = 0; a < 3; ++a) {
        g.ih[a] = 1.0 / sp[a];
        g.sp[a] = sp[a];
    }
    const cudaError_t e = launch_jacobian_any<T>(field, g, J, num_sms(), s);
    if (e != cudaSuccess) {
        cudaGetLastError();
        report(__LINE__, __func__, cudaGetErrorString(e));
        return DTB_ERR_CUDA;
    }
    return DTB_OK;
}

}  // namespace

extern "C" int dtb_jacobian_device_noalloc(int precision, int order, size_t nx, size_t ny, size_t nz, double dx,
                                           double dy, double dz, const void *field, void *J, void *stream) {
    disptools_clear_error();
    if (nx < 3 || ny < 3 || nz < 3 || nx >= (1u << 30) || ny >= (1u << 30) || nz >= (1u << 30)) {
        report(__LINE__, __func__, "every axis needs at least 3 voxels");
        return DTB_ERR_ARGUMENT;
    }
    if (!field || !J) {
        report(__LINE__, __func__, "null array");
        return DTB_ERR_ARGUMENT;
    }
    if (order != 4 && order != 2) {
        report(__LINE__, __func__, "order must be 4 or 2");
        return DTB_ERR_ARGUMENT;
    }
    if (!(dx > 0.0 && dy > 0.0 && dz > 0.0)) {
        report(__LINE__, __func__, "spacing must be positive");
        return DTB_ERR_ARGUMENT;
    }
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    if (precision == DTB_PRECISION_FP64)
        return jacobian_noalloc<double>(nx, ny, nz, dx, dy, dz, order, static_cast<const double *>(field),
                                        static_cast<double *>(J), s);
    if (precision == DTB_PRECISION_MIXED)
        return jacobian_noalloc<float>(nx, ny, nz, dx, dy, dz, order, static_cast<const float *>(field),
                                       static_cast<float *>(J), s);
    report(__LINE__, __func__, "invalid precision");
    return DTB_ERR_ARGUMENT;
}
