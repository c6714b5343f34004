// qp3d_internal.h -- shared definitions between the host API and the kernels.
//
// Device layout of one shot (all float32, row pitch ldy = ny rounded up to 32
// so every row starts on a 128-byte boundary):
//   U[3]            wavefields u(k-1), u(k), u(k+1), rotated by index: a step
//                   never overwrites its inputs
//   VP, E2, R8      per-cell parameters vp, 2*eps, 8*(eps-delta)
//   W1[3],W3[3],P[3] PML split fields, three time levels each, and W21[2],
//                   rotated by index (no copies).  These are full "shadow"
//                   volumes: only PML cells are ever touched, so a cell's
//                   state lives at the cell's own index whatever face owns it.
//   record          nt * hx * hy receiver samples
//   gmax            nt floats: max|grad u| of each step (bits, atomicMax)
#pragma once

#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include <vector>

namespace qp3d {

constexpr int kRadius = 5;        // 10th-order stencil (M/2 with M = 10)
constexpr int kTileY = 32;        // y cells per tile = 8 quads of 4 cells
constexpr int kQuadsY = kTileY / 4;
constexpr int kHaloY = 8;         // y halo rounded up to 16 bytes
constexpr int kBoxY = kTileY + 2 * kHaloY;   // 48 floats per staged halo row
// Load groups in flight or in use: the current plane's and those ahead.  The
// step kernels take microseconds a plane, so one ahead covers a load (a third
// group with 28-row tiles in the same memory made no difference); the gradmax
// kernels are done with a plane sooner than its load takes.
constexpr int kGroups = 2, kGradmaxGroups = 3;
// Tile height of the allocation-free maximum.  The kernel is bound by shared-
// memory bandwidth (25 16-byte loads a quad) and its latency; 24-row tiles
// leave room for four CTAs an SM: 460x460x360 278 us a call with 32 rows, 264
// with 24; 240x240x190 65 and 60.
constexpr int kGradmaxTileX = 24;
// own-cell planes staged
__host__ __device__ constexpr int ring_z(int groups) { return 2 * kRadius + groups; }
constexpr int kMaxTileX = 32;
constexpr int kThreads = kQuadsY * kMaxTileX;        // 256
constexpr int kStepTileX = 32;   // largest tile height of the step kernels
constexpr int kStepThreads = kQuadsY * kStepTileX;
constexpr int kMaxFusedSources = 64;
// Relative prediction errors of the step max kept for the speculative window
// (most recent first).
constexpr int kSpecHist = 8;
constexpr int kMaxPml = 256;
constexpr int kWinFloats = 5;

// The two tensor maps of a wavefield buffer: boxes of the tile's own cells and
// of the tile with its halo.
struct TileMaps {
    CUtensorMap z, c;
};

// Error bits written to the device error word.
constexpr unsigned kErrWaitTimeout = 1u;

struct Coefs {
    float cx[kRadius], cy[kRadius], cz[kRadius];      // c[31+m]/h
    float c2x[kRadius], c2y[kRadius], c2z[kRadius];   // c2[31+m]/h^2
    float kx, ky, kz;                                  // -2*sum(c2?)
    // the same values duplicated in both lanes, for the paired FP32x2 stencil
    float2 cx2[kRadius], cy2[kRadius], cz2[kRadius];
    float2 c2x2[kRadius], c2y2[kRadius], c2z2[kRadius];
    float2 kx2, ky2, kz2;
    // Reference arithmetic (qp3d_exact.h): the tables as given (both lanes
    // alike) and per axis the divisors of the first and second derivatives,
    // h and h*h rounded.
    float2 rc[kRadius], rc2[kRadius];                  // c[31+m], c2[31+m]
    float rh[3], rh2[3];                               // x, y, z
    // their rounded reciprocals, and whether weights and divisors allow the
    // division by them (xr::div_const)
    float ry[3], ry2[3];
    int div_ok;
};

// Arithmetic of the step: the reference CPU operators' roundings
// (qp3d_exact.h, bit-identical to CPU_function.c) or the folded fast form.
enum Arith { kArithRef = 0, kArithFast = 1 };

// One source sample: padded coordinates and the amplitude.
struct SrcEntry {
    int x, y, z;
    float v;
};

struct PlaneParams {
    // geometry
    int nx, ny, nz, ldy, pml, sz;
    int tile_x;          // rows per tile (<= kMaxTileX)
    int chunk_z;         // planes per z chunk
    long long plane;     // nx * ldy
    Coefs k;
    float dt;
    int step;            // time step index k
    float wavelet;       // wavelet[k]
    // wavefields: u(k) is staged by TMA (and read directly by the fix-up);
    // u(k-1) read, u(k+1) written
    const float *u_cur;
    const float *u_prev;
    float *u_out;
    const float *prm_v, *prm_e, *prm_r;   // vp, 2 eps, 8 (eps - delta)
    // half-precision parameter storage (half_params != 0): vp, eps, delta as
    // IEEE half, widened in the kernels; prm_* are unused then
    const __half *h_vp, *h_eps, *h_del;
    int half_params;
    const float *w1o, *w1c; float *w1n;   // w11, w12 -> w13
    const float *w3o, *w3c; float *w3n;   // w31, w32 -> w33
    const float *po, *pc; float *pn;      // p1, p2 -> p3
    const float *w21o; float *w21n;       // w21 -> w21'
    const float4 *layers;     // [3][pml] (a1h, a1l, d*dt, dd) for lr, fb, tb: the
                              // reference's a1 = (d*dt+1)^2 - 3 as an exact float
                              // pair; a2 = 2*d*dt - 1 and a3 = 1 - d*dt follow
    int arith;                // Arith of this launch
    float *gmax;              // gmax[0..nt): max|grad u| per step
    float *record;            // record plane of this step, or null
    const SrcEntry *src;      // sources inside the updated box, fused
    int nsrc;
    unsigned *err;
    // threshold decisions of the step, one bit per cell, 32 y cells a word
    // (word = pitched index / 32; FP32 parameters only): written to dec_out
    // (a speculative step's resolution clears the bits of the cells it fixes),
    // or read from dec_in instead of being taken (exact steps: the gradient's
    // recomputation replays the forward's)
    unsigned *dec_out;
    const unsigned *dec_in;
    unsigned long long wait_ns;   // limit of every bounded device wait (0: 2 s)
    int hold_plane;           // test hook: plane hold_plane - 1 of the first CTA is
                              // never loaded, so its waits run out (0: none)
    // threshold handling of the step kernel
    int spec;                 // 1: predicted window, own max, deferred cells
    const int *gate;          // spec: set to 1 by a column whose segment overflowed and by
                              // the resolution of a step that is re-run (null: not spec)
    float *win;               // spec: kWinFloats of the step: M_lo, M_hi, M_pred and the
                              // thresholds of m2 at M_lo and M_hi
    int win_ready;            // 1: all five are there already
    float *win_next;          // where the resolution leaves the next step's (or null)
    const float *spec_err;    // kSpecHist last relative prediction errors of the max
    float delta_min;          // smallest half-width of the window
    float spec_bias;          // relative shift of the window (test hook, 0)
    // Cells whose decision waits for the exact max of the step ("deferred"),
    // listed by the column that holds them in a segment of its own: pitched
    // index and m2, and what gives the cell its S = 1 results: u(k+1) with
    // S = 1 without the source, or of a PML cell the three derivative terms of
    // its update (its other inputs are still in place).
    uint2 *dkey;
    float4 *dval;
    unsigned *dcount;         // cells listed per column (grid launches)
    unsigned dcap;            // entries per segment (grid launches)
    unsigned *alt_count;      // &alt_count[step]: deferred cells
    // batched launches only
    int ucur;                 // index of u(k) among the shot's three buffers
    int active;               // 0 once the shot has run all its steps
};

// One shot of a batched run, as the host lays it out in device memory; the
// per-step PlaneParams are derived from it on the device
// (qp3d_batch_prepare_kernel), so a captured step can be replayed.
struct BatchShot {
    int nx, ny, nz, ldy, pml, sz, nt, hx, hy;
    long long plane;
    float dt, delta_min;
    float *U[3];
    const float *VP, *E2, *R8;
    float *W1[3], *W3[3], *P[3], *W21[2];
    const float4 *layers;
    float *gmax;
    float *record;
    const SrcEntry *src;
    int nsrc;
    const float *wavelet;     // nt samples
    float *win;               // kWinFloats * nt
    int *redo;                // nt
    unsigned *alt_count;      // nt
    float *spec_err;
    uint2 *dkey;              // deferred cells (see PlaneParams), all columns
    float4 *dval;
    float spec_bias;
    unsigned *err;
};

// A unit of work of a batched launch: one tile column of one shot.
struct WorkItem {
    int shot, tile_x, y0, x0, z0, z1;
    unsigned dcap, dbase;     // its segment of the shot's deferred-cell list
};

// Kernel arguments of the batched plane kernels.  The coefficient tables are
// shared by all shots of a batch (same spacing and FD tables).
struct BatchArgs {
    Coefs k;
    const PlaneParams *pp;    // per shot, the current step
    const TileMaps *tm;       // per shot three pairs of maps (one per u buffer)
    const WorkItem *work;
    int nwork;
    unsigned *dcount;         // deferred cells per work item
    int nshots;
    int *queue;               // next item of the re-run (zeroed by the prepare kernel)
    int arith;                // Arith of every shot of the batch
};

// One backward step of the adjoint (qp3d_adjoint.cu): the adjoint state of
// s^{k+1} (L*) to that of s^k (N*), with the scalar operator of step k frozen
// from u^k and the step's threshold.  C: coefficient fields of the
// transposed derivatives (x, y, z first; xx, yy, zz second).  The adjoint of
// u_prev is not kept: at a cell of the interior it is minus the adjoint of u
// of the step after, elsewhere zero.
struct AdjParams {
    int nx, ny, nz, ldy, pml, sz, hx, hy;
    long long plane;
    Coefs k;
    float dt;
    const float *u;                        // u^k
    const float *VP, *E2, *R8;             // vp, 2 eps, 8 (eps - delta)
    const float4 *layers;
    const float *T2;                       // threshold m2 of step k
    const unsigned *dec;                   // or its decisions, one bit per cell (null: T2)
    const float *resid;                    // record residual of step k (hx * hy)
    const float *resid_prev;               // and of step k + 1 (null: k is the last)
    const float *Lprev;                    // Lu of step k + 1 (zero for the last step)
    const float *Lu, *Lw1, *Lw1o, *Lp, *Lpo, *Lw21, *Lw3, *Lw3o;
    float *Nu, *Nw1, *Nw1o, *Np, *Npo, *Nw21, *Nw3, *Nw3o;
    float *C[6];
    float *gK, *gE, *gD;                   // gradient sums over the steps
    int live;                              // 1: S's dependence on grad u included
    int tile_x, chunk_z;                   // pass A's tiles
    unsigned *err;
    unsigned long long wait_ns;
};

// Tile height of pass A: with its 15 streams two CTAs of 24 rows fit an SM,
// 12 warps with up to 168 registers a thread.
constexpr int kAdjTileX = 24;
void plan_adjoint(AdjParams &a, int nsm);
// tm: u^k's maps for tiles of a.tile_x rows
cudaError_t launch_adjoint_step(const TileMaps &tm, const AdjParams &a, cudaStream_t stream);
cudaError_t launch_threshold(const float *gmax, float *T2, int n, cudaStream_t stream);
cudaError_t launch_residual(const float *rec, const float *dobs, float *r, long long n,
                            double *misfit, cudaStream_t stream);
cudaError_t launch_to_bf16(const float *a, __nv_bfloat16 *h, long long n, cudaStream_t stream);
cudaError_t launch_from_bf16(const __nv_bfloat16 *h, float *a, long long n, cudaStream_t stream);

// Launchers (qp3d_kernels.cu).  All enqueue on `stream` and return the
// launch error.
cudaError_t launch_gradmax(const TileMaps &tm, const PlaneParams &p, dim3 grid,
                           cudaStream_t stream);
cudaError_t launch_step(const TileMaps &tm, const PlaneParams &p, dim3 grid, size_t smem,
                        cudaStream_t stream);
// resolution of a speculative step: the fix-up of its deferred cells or (when
// the max fell outside the window or a segment overflowed) its exact re-run, a
// persistent grid of two CTAs an SM
cudaError_t launch_fix_or_rerun(const TileMaps &tm, const PlaneParams &p, float *spec_err,
                                int nsm, size_t smem, cudaStream_t stream);
cudaError_t launch_band_sources(float *u_new, const float *u_cur,
                                const SrcEntry *src, int n, long long plane,
                                int ldy, float w, cudaStream_t stream);
cudaError_t launch_all_sources(float *u_new, const float *u_cur,
                               const SrcEntry *src, int n, long long plane,
                               int ldy, int nx, int ny, int nz, float w,
                               cudaStream_t stream);
cudaError_t launch_record(const float *u, float *rec, int nx, int ny, int pml,
                          int sz, int ldy, long long plane,
                          cudaStream_t stream);
cudaError_t launch_crop(const float *u, float *out, int x0, int x1, int y0,
                        int y1, int z0, int z1, int ldy, long long plane,
                        cudaStream_t stream);
// Per-cell parameters vp, 2 eps, 8 (eps - delta), or vp, eps, delta as
// IEEE half (round to nearest even), from dense [nz][nx][ny] volumes (the
// caller's layout, copied to the device in one piece) into the pitched
// layout, row padding zero.
cudaError_t launch_params_dense(const float *vp, const float *eps, const float *del, float *VP,
                                float *E2, float *R8, int nx, int ny, int nz, int ldy,
                                cudaStream_t stream);
cudaError_t launch_to_half_dense(const float *a, __half *h, int nx, int ny, int nz, int ldy,
                                 cudaStream_t stream);
// Every non-zero sample of dense [nz][nx][ny] source volumes, of each in index
// order (z, then x, then y), scanned by several host threads.
struct SourceVolume {
    const float *s;
    int nx, ny, nz;
    std::vector<SrcEntry> *out;
};
void scan_source_volumes(const std::vector<SourceVolume> &vols);
void scan_source_volume(const float *s, int nx, int ny, int nz, std::vector<SrcEntry> &out);
// Dynamic shared memory of a step kernel; nsrc = fused sources of the shot
// (the per-CTA source list has room for all of them); and of a gradmax kernel.
size_t plane_smem_bytes(int tile_x, int pml, int nsrc);
size_t gradmax_smem_bytes(int tile_x);
// The tensor maps of a pitched [nz][nx][ldy] wavefield for tiles of tile_x
// rows (cuTensorMapEncodeTiled's result).
typedef CUresult (*EncodeTiledFn)(CUtensorMap *, CUtensorMapDataType, cuuint32_t, void *,
                                  const cuuint64_t *, const cuuint64_t *, const cuuint32_t *,
                                  const cuuint32_t *, CUtensorMapInterleave, CUtensorMapSwizzle,
                                  CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
inline CUresult encode_tile_maps(EncodeTiledFn encode, const float *base, int nx, int ny, int nz,
                                 int ldy, int tile_x, TileMaps *tm)
{
    cuuint64_t dims[3] = {(cuuint64_t)ny, (cuuint64_t)nx, (cuuint64_t)nz};
    cuuint64_t strides[2] = {(cuuint64_t)ldy * 4, (cuuint64_t)ldy * 4 * nx};
    cuuint32_t zbox[3] = {(cuuint32_t)kTileY, (cuuint32_t)tile_x, 1};
    cuuint32_t cbox[3] = {(cuuint32_t)kBoxY, (cuuint32_t)(tile_x + 2 * kRadius), 1};
    cuuint32_t es[3] = {1, 1, 1};
    CUresult r = CUDA_SUCCESS;
    for (int i = 0; i < 2 && r == CUDA_SUCCESS; ++i)
        r = encode(i ? &tm->c : &tm->z, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 3,
                   const_cast<float *>(base), dims, strides, i ? cbox : zbox, es,
                   CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE,
                   CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    return r;
}

// Batched launches.  kind: 0 gradmax, 1 exact step, 2 speculative step; the
// resolution of a speculative step runs on grid persistent CTAs.
size_t batch_smem_bytes(int tile_x, int pml, int nsrc);
cudaError_t launch_batch_prepare(const BatchShot *shots, int nshots, PlaneParams *pp, int *ctr,
                                 int *queue, int spec, cudaStream_t stream);
cudaError_t launch_batch_plane(int kind, const BatchArgs &b, int threads, size_t smem,
                               cudaStream_t stream);
cudaError_t launch_batch_resolve(const BatchArgs &b, int grid, int threads, size_t smem,
                                 cudaStream_t stream);
// max|grad u| in one launch: sc starts zero and is left zero, out receives the
// maximum (NaN on a timed-out wait) and *host_flags (mapped) the error bits.
struct alignas(64) GradmaxScratch {
    unsigned max_bits, done, err;
};
cudaError_t launch_gradmax_direct(const float *u, int nx, int ny, int nz, int ldy, const Coefs &k,
                                  int nsm, cudaStream_t stream, GradmaxScratch *sc, float *out,
                                  unsigned *host_flags);
// the same from TMA-staged planes
cudaError_t configure_gradmax_single();
cudaError_t launch_gradmax_single(const TileMaps &tm, const PlaneParams &p, dim3 grid,
                                  cudaStream_t stream, GradmaxScratch *sc, float *out,
                                  unsigned *host_flags);
// threads of a plane kernel's CTA: whole warps; rows past tile_x are idle, so
// every warp collective sees 32 lanes
__host__ __device__ inline int plane_threads(int tile_x) { return (kQuadsY * tile_x + 31) & ~31; }
// z chunks of a plane kernel's grid
int plan_chunks(long long tiles, int ncz, int threads, size_t smem, int nsm);
cudaError_t configure_kernels();

}  // namespace qp3d
