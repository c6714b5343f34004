// qp3d_noalloc.cu -- max|grad u| of a caller's device wavefield without any
// device allocation.
//
// Some callers cannot let a library allocate device memory: a host program
// whose framework has already reserved the whole device for its own pool, or
// a real-time loop that forbids allocation after start-up.
// qp3d_gradmax_noalloc serves them.  It has the arithmetic of the library's
// gradmax kernel, with its scratch (the maximum, a count of finished CTAs and an
// error word) in a file-scope device variable of this translation unit
// instead of buffers the library allocates; the caller passes the wavefield
// and the output location.  A call is one launch and one wait: the last CTA
// delivers the maximum and writes the error flags to mapped host memory
// (measured on 240x240x190: 90 us with a cleared error word, a second kernel
// over partial maxima and a copy of the flags).
//
// The scratch exists once per device that loads the library and is held until
// the process exits: kSlots entries, one for each call under way.  A call waits
// for its stream before it returns (so that a bounded device wait that ran out
// is reported as QP3D_ERR_TIMEOUT) and keeps its entry until then, so host
// threads may call at the same time; the last CTA leaves the entry zero for the
// next call.  (One entry for all: two calls whose kernels overlapped could each
// miss the last of its CTAs, and the count stayed wrong for the process.)
#include "qp3d.h"
#include "qp3d_internal.h"

#include <algorithm>
#include <condition_variable>
#include <cstdio>
#include <cstring>
#include <mutex>

namespace qp3d {
void derive_coefs(const float *c, const float *c2, float dx, float dy, float dz, Coefs *k);
}
using namespace qp3d;

namespace {

// Largest number of 32-cell x 32-row tiles per plane: nx*ny up to about 64 M
// cells.
constexpr unsigned kNoAllocMaxTiles = 1u << 16;

// 96 MB of the 129 MB L2
constexpr long long kDirectMaxCells = 24ll << 20;

constexpr int kSlots = 32;       // a bit each in DeviceScratch::busy
constexpr int kFlagStride = 16;  // a 64-byte line each
static __device__ GradmaxScratch g_noalloc_scratch[kSlots];

struct DeviceScratch {
    bool ready;
    GradmaxScratch *sc;
    unsigned *flags;      // mapped host words
    unsigned busy;
};
constexpr int kMaxDevices = 64;
DeviceScratch g_dev[kMaxDevices];
std::mutex g_mutex;
std::condition_variable g_slot_free;

// A call's entry of its device's scratch, from its launch to the end of its
// wait; with all of them taken the call waits for one.
struct Slot {
    DeviceScratch &d;
    int i = 0;
    explicit Slot(DeviceScratch &dev) : d(dev)
    {
        std::unique_lock<std::mutex> lock(g_mutex);
        g_slot_free.wait(lock, [&] { return d.busy != ~0u; });
        while (d.busy >> i & 1u) ++i;
        d.busy |= 1u << i;
    }
    ~Slot()
    {
        std::lock_guard<std::mutex> lock(g_mutex);
        d.busy &= ~(1u << i);
        g_slot_free.notify_all();
    }
    GradmaxScratch *scratch() const { return d.sc + i; }
    unsigned *flags() const { return d.flags + kFlagStride * i; }
};
static_assert(kSlots == 32, "one bit of busy each");

EncodeTiledFn g_encode = nullptr;

int report(char *err, size_t errlen, int code, const char *msg)
{
    if (err && errlen) snprintf(err, errlen, "%s", msg);
    return code;
}

// test hooks (set through qp3d_tune with a NULL context)
unsigned long long g_wait_ns = 0;   // 0: the kernels' default (2 s)
int g_hold_plane = 0;               // withheld plane + 1 in the first CTA, 0: none

}  // namespace

namespace qp3d {
int noalloc_tune(const char *key, int value)
{
    if (!strcmp(key, "noalloc_wait_limit_us") && value >= 0) g_wait_ns = 1000ull * (unsigned)value;
    else if (!strcmp(key, "noalloc_test_hold_plane") && value >= -1) g_hold_plane = value + 1;
    else return QP3D_ERR_ARG;
    return QP3D_OK;
}
}  // namespace qp3d

extern "C" int qp3d_gradmax_noalloc(const float *d_u, int nx, int ny, int nz, int ldy, float dx,
                                    float dy, float dz, const float *c, float *d_max,
                                    void *stream, char *err, size_t errlen)
{
    char msg[256];
    if (err && errlen) err[0] = 0;
    if (!d_u || !d_max || !c)
        return report(err, errlen, QP3D_ERR_ARG, "null wavefield, output or coefficient table");
    if (nx < 11 || ny < 11 || nz < 11)
        return report(err, errlen, QP3D_ERR_ARG, "grid smaller than 11 cells in some direction");
    if (ldy < ny || ldy % 4 != 0)
        return report(err, errlen, QP3D_ERR_ARG, "row pitch ldy must be >= ny and a multiple of 4");
    if (reinterpret_cast<uintptr_t>(d_u) % 16 != 0)
        return report(err, errlen, QP3D_ERR_ARG, "wavefield pointer must be 16-byte aligned");
    if (!(dx > 0) || !(dy > 0) || !(dz > 0))
        return report(err, errlen, QP3D_ERR_ARG, "non-positive spacing");

    int dev = 0, nsm = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kMaxDevices ||
        cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess)
        return report(err, errlen, QP3D_ERR_CUDA, "no usable CUDA device");

    // launch plan (as the shot path plans it)
    const int ncx = nx - 2 * kRadius, ncz = nz - 2 * kRadius;
    const int ntx = (ncx + kGradmaxTileX - 1) / kGradmaxTileX;
    const int tile_x = (ncx + ntx - 1) / ntx;
    const int nxt = (ncx + tile_x - 1) / tile_x;
    const int nyt = (ny - kRadius - 1) / kTileY + 1;
    const long long tiles = (long long)nxt * nyt;
    const int nxt32 = (ncx + 31) / 32;
    const long long tiles32 = (long long)nxt32 * nyt;
    if (tiles32 > kNoAllocMaxTiles) {
        snprintf(msg, sizeof(msg),
                 "grid %dx%d needs %lld tiles per z chunk; qp3d_gradmax_noalloc holds at most %u",
                 nx, ny, tiles32, kNoAllocMaxTiles);
        return report(err, errlen, QP3D_ERR_ARG, msg);
    }
    long long nch = plan_chunks(tiles, ncz, plane_threads(tile_x), gradmax_smem_bytes(tile_x), nsm);
    const int chunk_z = (int)((ncz + nch - 1) / nch);
    nch = (ncz + chunk_z - 1) / chunk_z;
    // the documented limits, in tiles of 32 x 32 cells and z chunks (the launch
    // grid is (tiles of a plane, 1, z chunks), and CUDA limits its third
    // dimension to 65535)
    if (nxt32 > 65535 || nch > 65535) {
        snprintf(msg, sizeof(msg),
                 "grid %dx%dx%d needs %d x tiles and %lld z chunks; a call takes at most 65535",
                 nx, ny, nz, nxt32, nch);
        return report(err, errlen, QP3D_ERR_ARG, msg);
    }

    // once per device, with that device current: the scratch addresses and
    // the kernel's shared-memory limit.  The first call on a device does this
    // set-up; make it before any stream capture.
    {
        std::lock_guard<std::mutex> lock(g_mutex);
        if (!g_encode) {
            void *fn = nullptr;
            cudaDriverEntryPointQueryResult qr;
            if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &fn, 12000,
                                                 cudaEnableDefault, &qr) != cudaSuccess ||
                qr != cudaDriverEntryPointSuccess || !fn)
                return report(err, errlen, QP3D_ERR_CUDA, "cuTensorMapEncodeTiled unavailable");
            g_encode = reinterpret_cast<EncodeTiledFn>(fn);
        }
        DeviceScratch &d = g_dev[dev];
        if (!d.ready) {
            GradmaxScratch *sc = nullptr;
            unsigned *flags = nullptr;
            if (cudaGetSymbolAddress((void **)&sc, g_noalloc_scratch) != cudaSuccess || !sc)
                return report(err, errlen, QP3D_ERR_CUDA, "cudaGetSymbolAddress failed");
            if (configure_gradmax_single() != cudaSuccess)
                return report(err, errlen, QP3D_ERR_CUDA, "cannot set the kernel's shared memory");
            if (cudaHostAlloc((void **)&flags, kSlots * kFlagStride * sizeof(unsigned),
                              cudaHostAllocMapped | cudaHostAllocPortable) != cudaSuccess)
                return report(err, errlen, QP3D_ERR_NOMEM, "cannot allocate the host flag words");
            d.sc = sc;
            d.flags = flags;
            d.ready = true;
        }
    }

    // Through L1 as long as the volume stays in L2, from staged planes beyond,
    // where their loads ahead of use pay.  Calls in a loop, through L1 and staged:
    // 240x240x190 (11 Mi cells) 42 and 56 us, 300x300x200 (18) 63 and 80,
    // 300x300x262 (24) 99 and 99, 320x320x260 (25) 107 and 103, 400x400x300 (48)
    // 185 and 173, 460x460x360 (76) 271 and 259.  (With L2 full of other data the
    // two are closer, staged ahead: 65 and 63, 97 and 87, 121 and 105.)  The hook
    // that withholds a plane is the staged form's.
    const bool direct = (long long)nx * ldy * nz <= kDirectMaxCells && g_hold_plane == 0;
    TileMaps tm{};
    if (!direct) {   // the tensor maps of the staged form
        CUresult cr = encode_tile_maps(g_encode, d_u, nx, ny, nz, ldy, tile_x, &tm);
        if (cr == CUDA_ERROR_INVALID_CONTEXT) {   // a host thread that has used no CUDA yet
            (void)cudaFree(nullptr);              // gives it the device's context
            cr = encode_tile_maps(g_encode, d_u, nx, ny, nz, ldy, tile_x, &tm);
        }
        if (cr != CUDA_SUCCESS)
            return report(err, errlen, QP3D_ERR_CUDA, "cuTensorMapEncodeTiled failed");
    }

    PlaneParams p;
    memset(&p, 0, sizeof(p));
    p.nx = nx; p.ny = ny; p.nz = nz; p.ldy = ldy; p.pml = 0; p.sz = 0;
    p.tile_x = tile_x;
    p.chunk_z = chunk_z;
    p.plane = (long long)nx * ldy;
    derive_coefs(c, c, dx, dy, dz, &p.k);   // first-derivative weights only
    p.arith = kArithFast;   // the library's default arithmetic
    const Slot slot(g_dev[dev]);
    p.err = &slot.scratch()->err;
    p.wait_ns = g_wait_ns;
    p.hold_plane = g_hold_plane;
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    dim3 grid((unsigned)tiles, 1, (unsigned)nch);
    cudaError_t e = direct
        ? launch_gradmax_direct(d_u, nx, ny, nz, ldy, p.k, nsm, s, slot.scratch(), d_max,
                                slot.flags())
        : launch_gradmax_single(tm, p, grid, s, slot.scratch(), d_max, slot.flags());
    if (e != cudaSuccess) {
        snprintf(msg, sizeof(msg), "launch failed: %s", cudaGetErrorString(e));
        return report(err, errlen, QP3D_ERR_CUDA, msg);
    }
    // wait for the result and report a device wait that ran out (d_max then
    // holds NaN)
    if ((e = cudaStreamSynchronize(s)) != cudaSuccess) {
        snprintf(msg, sizeof(msg), "%s", cudaGetErrorString(e));
        return report(err, errlen, QP3D_ERR_CUDA, msg);
    }
    const unsigned flags = *const_cast<volatile unsigned *>(slot.flags());
    if (flags) return report(err, errlen, QP3D_ERR_TIMEOUT, "a device wait timed out");
    return QP3D_OK;
}
