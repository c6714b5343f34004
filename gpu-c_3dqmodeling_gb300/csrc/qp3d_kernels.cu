// qp3d_kernels.cu -- sm_103a kernels for the 3D pure-qP VTI time step.
//
// One time step of the reference (3dPureqPModeling_single_shot.cu:282-320:
// grad -> D2H + host absMaxval -> scalar_operator -> wavefield_update ->
// addsource -> exchange -> D2H + record crop) becomes:
//
//   qp3d_step_kernel      everything in one pass: gradient, scalar operator S
//                         (GPU_kernel.cu:87-115), Laplacians, interior
//                         leapfrog and the six split-field PML faces
//                         (GPU_kernel.cu:534-639), source injection
//                         (GPU_kernel.cu:720-731), the receiver plane
//                         (3dPureqPModeling_single_shot.cu:333-337), and the
//                         step's own max|grad u| (atomicMax on the float bits:
//                         all values are >= 0, so bit order is value order).
//                         The time-level rotation (GPU_kernel.cu:733-812) is
//                         done by the host swapping buffer indices.
//   the threshold         S needs the max of the step before any cell is
//                         updated: either qp3d_gradmax_kernel computes it
//                         first (GPU_kernel.cu:14-33 + CPU_function.c:10-22),
//                         or the step runs speculatively with a predicted
//                         window and qp3d_fix_or_rerun_kernel settles the
//                         cells whose decision waited (an exact re-run when
//                         the prediction missed).
//
// The same tile bodies run in the batched kernels (many shots per launch),
// and the adjoint kernels at the end of the file transpose the step.
//
// Both kernels march along z.  A CTA owns a tile of tile_x rows (x) by 32
// cells (y) and a chunk of z planes.  Each thread owns one row and four
// consecutive y cells (a "quad", one float4).  Planes of u(k) are staged by
// TMA (cp.async.bulk.tensor.3d) into two rings in shared memory, the tile's
// own cells for the z taps and the current plane with its halo for the x and
// y taps (see Pipe); the stencil reads all 30 taps from shared memory.
//
// What bounds the step: instruction issue and its latencies at 16 warps an SM
// (128 registers a thread), beside HBM on large grids.  Instructions per warp
// and plane (four rows by 32 cells; 240x240x190 cells, 20-cell shell) went
// from 764 to 652, 582 on a grid with a 6-cell shell, of which the stencil is
// 240: the shell's update has a loop body of its own, per axis and in FP32x2
// pairs; the threshold decides warps before cells; deferred cells are listed
// on the side; the sources and the receiver plane are handled after the loop.
// 460x460x360: 623 -> 531 us a step kernel (75% of the DRAM peak by ncu).
//
// Arithmetic.  The 1/h factors of the reference (each tap divided by dx or
// dx*dx, CPU_function.c:314-316,393-395) are folded into the coefficient
// tables, and a*b+c is fused where written as fmaf().  This translation unit
// is compiled with -fmad=false so that no other fusion happens: the result is
// bit-identical to the mirror variant of the CPU oracle.  The division of the
// scalar operator is a Newton-Raphson reciprocal (rcp_nr2: fused
// multiply-adds only, so the oracle reproduces it exactly); the square root
// is IEEE (sqrt.rn).
#include "qp3d_internal.h"
#include "qp3d_exact.h"

#include <math.h>

#include <algorithm>
#include <type_traits>

namespace qp3d {

// ---------------------------------------------------------------------------
// PTX helpers: mbarrier + TMA
// ---------------------------------------------------------------------------
__device__ __forceinline__ unsigned smem_u32(const void *p)
{
    return static_cast<unsigned>(__cvta_generic_to_shared(p));
}

__device__ __forceinline__ void mbar_init(uint64_t *bar, unsigned count)
{
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count)
                 : "memory");
}

__device__ __forceinline__ void mbar_arrive_expect_tx(uint64_t *bar, unsigned bytes)
{
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)),
                 "r"(bytes)
                 : "memory");
}

__device__ __forceinline__ bool mbar_try_wait(uint64_t *bar, unsigned parity)
{
    unsigned ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(smem_u32(bar)), "r"(parity)
        : "memory");
    return ok != 0;
}

__device__ __forceinline__ unsigned long long global_ns()
{
    unsigned long long t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}

// Bounded wait: gives up after limit_ns of wall time.
__device__ __forceinline__ bool mbar_wait_bounded(uint64_t *bar, unsigned parity,
                                                  unsigned long long limit_ns)
{
    if (mbar_try_wait(bar, parity)) return true;
    unsigned long long t0 = global_ns();
    for (;;) {
        if (mbar_try_wait(bar, parity)) return true;
        if (global_ns() - t0 > limit_ns) return false;
    }
}

__device__ __forceinline__ void fence_barrier_init()
{
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}

__device__ __forceinline__ void fence_proxy_async()
{
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
}

__device__ __forceinline__ void tma_load_3d(void *dst, const CUtensorMap *tm, int c0, int c1,
                                            int c2, uint64_t *bar)
{
    asm volatile(
        "cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes"
        " [%0], [%1, {%2, %3, %4}], [%5];" ::"r"(smem_u32(dst)),
        "l"(reinterpret_cast<uint64_t>(tm)), "r"(c0), "r"(c1), "r"(c2), "r"(smem_u32(bar))
        : "memory");
}

// 16 (8) bytes global -> shared, past L1, for the thread's own use after
// cp_async_wait
__device__ __forceinline__ void cp_async16(void *dst, const void *src)
{
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_u32(dst)), "l"(src)
                 : "memory");
}
__device__ __forceinline__ void cp_async8(void *dst, const void *src)
{
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(smem_u32(dst)), "l"(src)
                 : "memory");
}
__device__ __forceinline__ void cp_async_wait()
{
    asm volatile("cp.async.wait_all;" ::: "memory");
}

// Programmatic dependent launch: the kernels of a time step are launched with
// cudaLaunchAttributeProgrammaticStreamSerialization.  Each lets its successor
// start as soon as its own CTAs have, and waits for its predecessor to finish
// before it touches anything a step writes; what comes before the wait may
// only read data that no step changes.
__device__ __forceinline__ void pdl_trigger()
{
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

__device__ __forceinline__ float4 lds4(const float *p)
{
    return *reinterpret_cast<const float4 *>(p);
}

__device__ __forceinline__ float f4(const float4 &v, int j)
{
    return j == 0 ? v.x : j == 1 ? v.y : j == 2 ? v.z : v.w;
}

// ---------------------------------------------------------------------------
// Shared-memory layout of the plane kernels
// ---------------------------------------------------------------------------
struct SmemLayout {
    int zslot, cslot;     // floats of one own-cell plane and one halo plane
    size_t c_off;         // halo planes (the own-cell planes start at 0)
    size_t own_off;       // per-thread stream slots (step kernels)
    size_t bar_off;       // kGroups mbarriers
    size_t cnt_off;       // kGroups arrival counters, then the issued count
    size_t tab_off;       // layer coefficients: [3][pml] float4 (x, y, z faces)
    size_t ytab_off;      // those of the tile's y cells, [4][kTileY] floats
    size_t src_off;       // fused source entries of this CTA
    size_t misc_off;      // scalars
    size_t total;
};

// streams: 16-byte slots per thread (0 for the gradmax kernels)
__host__ __device__ inline SmemLayout smem_layout(int tile_x, int pml, int nsrc, int streams,
                                                  int groups = kGroups)
{
    SmemLayout L;
    L.zslot = tile_x * kTileY;
    L.cslot = ((tile_x + 2 * kRadius) * kBoxY + 31) & ~31;
    L.c_off = (size_t)L.zslot * 4 * ring_z(groups);
    L.own_off = L.c_off + (size_t)L.cslot * 4 * groups;
    L.bar_off = L.own_off + (size_t)plane_threads(tile_x) * 16 * streams;
    L.cnt_off = L.bar_off + 8 * groups;
    L.tab_off = (L.cnt_off + 4 * (groups + 1) + 15) & ~(size_t)15;
    L.ytab_off = L.tab_off + (streams ? 16 * 3 * (size_t)(pml > 0 ? pml : 1) : 0);
    L.src_off = L.ytab_off + (streams ? 16 * kTileY : 0);
    L.misc_off = L.src_off + (streams ? sizeof(SrcEntry) * (size_t)(nsrc > 0 ? nsrc : 1) : 0);
    L.misc_off = (L.misc_off + 15) & ~(size_t)15;
    L.total = L.misc_off + 64;
    return L;
}

// Streams of the step kernels: u(k-1), vp, 2 eps, 8 (eps - delta), and where
// there is a PML shell the seven split-field values a PML cell reads.
__host__ __device__ inline int step_streams(int pml) { return pml > 0 ? 11 : 4; }

size_t plane_smem_bytes(int tile_x, int pml, int nsrc)
{
    return smem_layout(tile_x, pml, nsrc, step_streams(pml)).total;
}

size_t gradmax_smem_bytes(int tile_x)
{
    return smem_layout(tile_x, 0, 0, 0, kGradmaxGroups).total;
}

// The number of z chunks of a plane kernel's grid: tiles columns of ncz planes,
// smem bytes a CTA.  A CTA's march over its planes is a serial chain (2-3 us a
// plane when two CTAs share an SM), so a grid too small to fill the SMs takes
// as long as its longest chunk, and one that fills them a little more than
// once takes two of them.  The estimate below, in planes, follows what was
// measured on 140^3, 191x127x105, 240x240x190 and 460x460x360 cells over 4 to
// 26 chunks: half-filled SMs run a plane 0.7 times as long; up to one wave
// costs its chunk and 1.5 planes of start-up; more waves overlap, at half a
// plane each and a third of a wave for the uneven end; the last factor is the
// re-read of ten planes a chunk.  Before (24 planes or more a chunk, 18 CTAs
// an SM) 140^3 took 63 us a step, now 43.
int plan_chunks(long long tiles, int ncz, int threads, size_t smem, int nsm)
{
    const int per_sm = std::max(1, std::min((int)(227 * 1024 / (smem + 1024)), 512 / threads));
    const double slots = (double)per_sm * nsm;
    int best = 1;
    double best_t = 0.0;
    for (int n = 1; n <= ncz && (n == 1 || tiles * n <= 64 * (long long)slots); ++n) {
        const int chunk = (ncz + n - 1) / n;
        if ((ncz + chunk - 1) / chunk != n) continue;   // the same chunks with fewer
        const double w = (double)tiles * n / slots;
        const double waves = w <= 0.5 ? 0.7 : (w <= 1.0 ? 1.0 : w + 0.35);
        const double t = waves * (chunk + (w <= 1.0 ? 1.5 : 0.5)) * (1.0 + 0.5 / chunk);
        if (n == 1 || t < best_t) {
            best = n;
            best_t = t;
        }
    }
    return best;
}

// ---------------------------------------------------------------------------
// Threshold of the scalar operator, GPU_kernel.cu:99.
//   (double)mode > 1.0e-02 * uxyzMax  <=>  mode > Tf, Tf = largest float not
//   above the double product;  mode = sqrtf(m2) > Tf  <=>  m2 > T2 with
//   T2 = max{x : sqrtf(x) <= Tf}.  The oracle derives T2 the same way.
// ---------------------------------------------------------------------------
__device__ float threshold_m2(float gmax)
{
    double td = 1.0e-02 * (double)gmax;
    float t = __double2float_rd(td);
    if (!(t >= 0.0f)) return t;
    float x = __fmul_rn(t, t);
    for (int it = 0; it < 64 && x > 0.0f && __fsqrt_rn(x) > t; ++it) x = nextafterf(x, 0.0f);
    for (int it = 0; it < 64; ++it) {
        float n = nextafterf(x, INFINITY);
        if (isinf(n) || __fsqrt_rn(n) > t) break;
        x = n;
    }
    return x;
}

// ---------------------------------------------------------------------------
// Stencil over one quad: first and second derivatives along x, y, z of the
// four cells (x, y..y+3, z) from the staged planes.  Cells (0,1) and (2,3)
// are processed as pairs with the packed FP32x2 instructions (add/mul/fma
// .rn.f32x2, round-to-nearest per lane, so every lane is bit-identical to
// the scalar operation it replaces).
// ---------------------------------------------------------------------------
__device__ __forceinline__ float2 f2(float a, float b) { return make_float2(a, b); }
__device__ __forceinline__ float2 sub2(float2 a, float2 b)
{
    return __fadd2_rn(a, make_float2(-b.x, -b.y));
}

__device__ __forceinline__ float2 half2of(const float4 &v, int h)
{
    return h ? make_float2(v.z, v.w) : make_float2(v.x, v.y);
}

// One second-difference tap in the reference's form, (u[+m] - 2u) + u[-m]
// (CPU_function.c:393-395), two cells at a time.  Summing c2[m] times these
// keeps a constant field's Laplacian exactly zero; the form with the centre
// weight folded into one coefficient, -2 sum(c2[m]) u + sum c2[m](u[+m] +
// u[-m]), does not (its rounded coefficients leave a term proportional to u),
// and that systematic term grew to 1.6e-5 relative L2 against the reference
// arithmetic over a 1000-step shot, against 6.7e-6 with this form.
__device__ __forceinline__ float2 lap_tap2(float2 a, float2 b, float2 u0)
{
    return __fadd2_rn(__ffma2_rn(make_float2(-2.0f, -2.0f), u0, a), b);
}

// Where a quad finds its taps: pc, its first cell in the halo plane of the
// current z (x and y taps), and za, its first cell in the own-cell plane z - 5
// (z taps); the planes after it follow at zslot floats each, those past the
// last slot (from the wrap-th on) one ring length (zlen) back.
struct Taps {
    const float *pc, *za;
    int wrap, zslot, zlen;
};

__device__ __forceinline__ float4 ztap(const Taps &T, int j)   // plane z - 5 + j
{
    return lds4((j < T.wrap ? T.za : T.za - T.zlen) + j * T.zslot);
}

template <bool SECOND>
__device__ __forceinline__ void quad_derivs(const Taps &T, const Coefs &k, float Ux[4],
                                            float Uy[4], float Uz[4], float Uxx[4], float Uyy[4],
                                            float Uzz[4], float u0[4])
{
    const float *pc = T.pc;
    // y taps: columns c-8 .. c+11 of the centre plane
    float Y[20];
#pragma unroll
    for (int b = 0; b < 5; ++b) {
        float4 v = lds4(pc - 8 + 4 * b);
        Y[4 * b] = v.x; Y[4 * b + 1] = v.y; Y[4 * b + 2] = v.z; Y[4 * b + 3] = v.w;
    }
#pragma unroll
    for (int h = 0; h < 2; ++h) {
        const int j0 = 2 * h, j1 = 2 * h + 1;
        const float2 c0 = f2(Y[8 + j0], Y[8 + j1]);
        u0[j0] = c0.x;
        u0[j1] = c0.y;
        float2 g = f2(0.0f, 0.0f), l = f2(0.0f, 0.0f);
#pragma unroll
        for (int m = 0; m < kRadius; ++m) {
            const float2 a = f2(Y[8 + j0 + m + 1], Y[8 + j1 + m + 1]);
            const float2 b = f2(Y[8 + j0 - m - 1], Y[8 + j1 - m - 1]);
            const float2 d = sub2(a, b);
            g = (m == 0) ? __fmul2_rn(k.cy2[0], d) : __ffma2_rn(k.cy2[m], d, g);
            if (SECOND) l = (m == 0) ? __fmul2_rn(k.c2y2[0], lap_tap2(a, b, c0))
                                     : __ffma2_rn(k.c2y2[m], lap_tap2(a, b, c0), l);
        }
        Uy[j0] = g.x; Uy[j1] = g.y;
        if (SECOND) { Uyy[j0] = l.x; Uyy[j1] = l.y; }
    }
    // x taps: rows r +- m of the centre plane
    const float2 uc[2] = {f2(u0[0], u0[1]), f2(u0[2], u0[3])};
    float2 gx[2] = {f2(0.f, 0.f), f2(0.f, 0.f)}, lx[2] = {f2(0.f, 0.f), f2(0.f, 0.f)};
#pragma unroll
    for (int m = 0; m < kRadius; ++m) {
        const float4 a = lds4(pc + (m + 1) * kBoxY);
        const float4 b = lds4(pc - (m + 1) * kBoxY);
        const float2 a2[2] = {f2(a.x, a.y), f2(a.z, a.w)}, b2[2] = {f2(b.x, b.y), f2(b.z, b.w)};
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const float2 d = sub2(a2[h], b2[h]);
            gx[h] = (m == 0) ? __fmul2_rn(k.cx2[0], d) : __ffma2_rn(k.cx2[m], d, gx[h]);
            if (SECOND) lx[h] = (m == 0) ? __fmul2_rn(k.c2x2[0], lap_tap2(a2[h], b2[h], uc[h]))
                                         : __ffma2_rn(k.c2x2[m], lap_tap2(a2[h], b2[h], uc[h]),
                                                      lx[h]);
        }
    }
    Ux[0] = gx[0].x; Ux[1] = gx[0].y; Ux[2] = gx[1].x; Ux[3] = gx[1].y;
    if (SECOND) { Uxx[0] = lx[0].x; Uxx[1] = lx[0].y; Uxx[2] = lx[1].x; Uxx[3] = lx[1].y; }
    // z taps
    float2 gz[2] = {f2(0.f, 0.f), f2(0.f, 0.f)}, lz[2] = {f2(0.f, 0.f), f2(0.f, 0.f)};
#pragma unroll
    for (int m = 0; m < kRadius; ++m) {
        const float4 a = ztap(T, kRadius + m + 1);
        const float4 b = ztap(T, kRadius - m - 1);
        const float2 a2[2] = {f2(a.x, a.y), f2(a.z, a.w)}, b2[2] = {f2(b.x, b.y), f2(b.z, b.w)};
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const float2 d = sub2(a2[h], b2[h]);
            gz[h] = (m == 0) ? __fmul2_rn(k.cz2[0], d) : __ffma2_rn(k.cz2[m], d, gz[h]);
            if (SECOND) lz[h] = (m == 0) ? __fmul2_rn(k.c2z2[0], lap_tap2(a2[h], b2[h], uc[h]))
                                         : __ffma2_rn(k.c2z2[m], lap_tap2(a2[h], b2[h], uc[h]),
                                                      lz[h]);
        }
    }
    Uz[0] = gz[0].x; Uz[1] = gz[0].y; Uz[2] = gz[1].x; Uz[3] = gz[1].y;
    if (SECOND) { Uzz[0] = lz[0].x; Uzz[1] = lz[0].y; Uzz[2] = lz[1].x; Uzz[3] = lz[1].y; }
}

// ---------------------------------------------------------------------------
// The same derivatives in the reference's arithmetic (CPU_function.c:314-316,
// 393-395; qp3d_exact.h): per tap c*(u[+m]-u[-m]) / h and
// c2*((u[+m]-2u) + u[-m]) / h^2, each operation rounded, IEEE division, the
// taps summed in order from 0.  Products and sums two cells at a time with
// the packed FP32x2 instructions.
// ---------------------------------------------------------------------------
__device__ __forceinline__ float2 div2(float2 p, float h)
{
    return make_float2(__fdiv_rn(p.x, h), __fdiv_rn(p.y, h));
}

// How the taps divide: IEEE division, or xr::div_const or
// xr::div_const_scaled in packed form.  IEEE divisions, with their slow path
// for the subnormal values ahead of a wavefront, were 9300 of the instructions
// a warp spent on a plane (998 us a step on 140^3; 223 with products in their
// place; 298 with the two forms below).
enum TapDiv { kDivIeee, kDivConst, kDivScaled };

__device__ __forceinline__ float2 div_const2(float2 p, float h, float y)
{
    const float2 nh = make_float2(-h, -h), y2 = make_float2(y, y);
    const float2 q0 = __fmul2_rn(p, y2);
    const float2 q1 = __ffma2_rn(__ffma2_rn(q0, nh, p), y2, q0);
    return __ffma2_rn(__ffma2_rn(q1, nh, p), y2, q1);
}

template <int DIV>
__device__ __forceinline__ float2 tap_div2(float2 p, float h, float y)
{
    if (DIV == kDivIeee) return div2(p, h);
    if (DIV == kDivConst) return div_const2(p, h, y);
    const float up = 18446744073709551616.0f, down = 5.4210109e-20f;   // 2^64, 2^-64
    const float half = 1.2924697e-26f, grid = 1.4012985e-45f;          // 2^-86, 2^-149
    const float2 ps = __fmul2_rn(p, make_float2(up, up));
    const float2 q = div_const2(ps, h, y);
    const float2 r = __ffma2_rn(q, make_float2(-h, -h), ps);
    float2 t = __fmul2_rn(q, make_float2(down, down));
    const float2 e = __ffma2_rn(t, make_float2(-up, -up), q);
    if (fabsf(e.x) == half && (e.x > 0.0f ? r.x > 0.0f : r.x < 0.0f))
        t.x = __fadd_rn(t.x, copysignf(grid, e.x));
    if (fabsf(e.y) == half && (e.y > 0.0f ? r.y > 0.0f : r.y < 0.0f))
        t.y = __fadd_rn(t.y, copysignf(grid, e.y));
    return t;
}

// one tap (m) of both derivatives along an axis for a pair of cells: a = u[+m],
// b = u[-m]
template <int DIV>
__device__ __forceinline__ void tap2(float2 a, float2 b, float2 u0, const Coefs &k, int m, int ax,
                                     float2 &g, float2 &l)
{
    g = __fadd2_rn(g, tap_div2<DIV>(__fmul2_rn(k.rc[m], sub2(a, b)), k.rh[ax], k.ry[ax]));
    l = __fadd2_rn(l, tap_div2<DIV>(__fmul2_rn(k.rc2[m], lap_tap2(a, b, u0)), k.rh2[ax], k.ry2[ax]));
}

__device__ __forceinline__ void quad_derivs_ref(const Taps &T, const Coefs &k, float Ux[4],
                                                float Uy[4], float Uz[4], float Uxx[4],
                                                float Uyy[4], float Uzz[4], float u0[4])
{
    const float *pc = T.pc;
    const float2 zero = make_float2(0.0f, 0.0f);
    float Y[20];
#pragma unroll
    for (int b = 0; b < 5; ++b) {
        float4 v = lds4(pc - 8 + 4 * b);
        Y[4 * b] = v.x; Y[4 * b + 1] = v.y; Y[4 * b + 2] = v.z; Y[4 * b + 3] = v.w;
    }
    float2 c0[2];
#pragma unroll
    for (int h = 0; h < 2; ++h) {
        const int j0 = 2 * h, j1 = 2 * h + 1;
        c0[h] = f2(Y[8 + j0], Y[8 + j1]);
        u0[j0] = c0[h].x;
        u0[j1] = c0[h].y;
        float2 g = zero, l = zero;
#pragma unroll
        for (int m = 0; m < kRadius; ++m)
            tap2<kDivConst>(f2(Y[8 + j0 + m + 1], Y[8 + j1 + m + 1]),
                       f2(Y[8 + j0 - m - 1], Y[8 + j1 - m - 1]), c0[h], k, m, 1, g, l);
        Uy[j0] = g.x; Uy[j1] = g.y;
        Uyy[j0] = l.x; Uyy[j1] = l.y;
    }
    float2 gx[2] = {zero, zero}, lx[2] = {zero, zero};
#pragma unroll
    for (int m = 0; m < kRadius; ++m) {
        const float4 a = lds4(pc + (m + 1) * kBoxY);
        const float4 b = lds4(pc - (m + 1) * kBoxY);
        const float2 a2[2] = {f2(a.x, a.y), f2(a.z, a.w)}, b2[2] = {f2(b.x, b.y), f2(b.z, b.w)};
#pragma unroll
        for (int h = 0; h < 2; ++h)
            tap2<kDivConst>(a2[h], b2[h], c0[h], k, m, 0, gx[h], lx[h]);
    }
    Ux[0] = gx[0].x; Ux[1] = gx[0].y; Ux[2] = gx[1].x; Ux[3] = gx[1].y;
    Uxx[0] = lx[0].x; Uxx[1] = lx[0].y; Uxx[2] = lx[1].x; Uxx[3] = lx[1].y;
    float2 gz[2] = {zero, zero}, lz[2] = {zero, zero};
#pragma unroll
    for (int m = 0; m < kRadius; ++m) {
        const float4 a = ztap(T, kRadius + m + 1);
        const float4 b = ztap(T, kRadius - m - 1);
        const float2 a2[2] = {f2(a.x, a.y), f2(a.z, a.w)}, b2[2] = {f2(b.x, b.y), f2(b.z, b.w)};
#pragma unroll
        for (int h = 0; h < 2; ++h)
            tap2<kDivConst>(a2[h], b2[h], c0[h], k, m, 2, gz[h], lz[h]);
    }
    Uz[0] = gz[0].x; Uz[1] = gz[0].y; Uz[2] = gz[1].x; Uz[3] = gz[1].y;
    Uzz[0] = lz[0].x; Uzz[1] = lz[0].y; Uzz[2] = lz[1].x; Uzz[3] = lz[1].y;
}

// The same with the other two divisions, as loops: they run for the warps
// around the leading edge of a wavefield, and three unrolled forms would not
// stay in the instruction cache.
template <int DIV>
__device__ __forceinline__ void quad_derivs_ref_loop(const Taps &T, const Coefs &k, float Ux[4],
                                                     float Uy[4], float Uz[4], float Uxx[4],
                                                     float Uyy[4], float Uzz[4], float u0[4])
{
    const float4 c = lds4(T.pc);
    const float2 c0[2] = {f2(c.x, c.y), f2(c.z, c.w)};
    u0[0] = c.x; u0[1] = c.y; u0[2] = c.z; u0[3] = c.w;
    float2 g[3][2], l[3][2];
#pragma unroll
    for (int ax = 0; ax < 3; ++ax) {
        g[ax][0] = g[ax][1] = l[ax][0] = l[ax][1] = make_float2(0.0f, 0.0f);
#pragma unroll 1
        for (int m = 0; m < kRadius; ++m) {
            float4 a, b;
            if (ax == 0) {
                a = lds4(T.pc + (m + 1) * kBoxY);
                b = lds4(T.pc - (m + 1) * kBoxY);
            } else if (ax == 1) {
                const float *pa = T.pc + m + 1, *pb = T.pc - m - 1;
                a = make_float4(pa[0], pa[1], pa[2], pa[3]);
                b = make_float4(pb[0], pb[1], pb[2], pb[3]);
            } else {
                a = ztap(T, kRadius + m + 1);
                b = ztap(T, kRadius - m - 1);
            }
            tap2<DIV>(f2(a.x, a.y), f2(b.x, b.y), c0[0], k, m, ax, g[ax][0], l[ax][0]);
            tap2<DIV>(f2(a.z, a.w), f2(b.z, b.w), c0[1], k, m, ax, g[ax][1], l[ax][1]);
        }
    }
#pragma unroll
    for (int h = 0; h < 2; ++h) {
        Ux[2 * h] = g[0][h].x; Ux[2 * h + 1] = g[0][h].y;
        Uy[2 * h] = g[1][h].x; Uy[2 * h + 1] = g[1][h].y;
        Uz[2 * h] = g[2][h].x; Uz[2 * h + 1] = g[2][h].y;
        Uxx[2 * h] = l[0][h].x; Uxx[2 * h + 1] = l[0][h].y;
        Uyy[2 * h] = l[1][h].x; Uyy[2 * h + 1] = l[1][h].y;
        Uzz[2 * h] = l[2][h].x; Uzz[2 * h + 1] = l[2][h].y;
    }
}

// What four wavefield values ask of the division: 0 when each is 0 or in
// [kWinLo, kWinHi], bit 0 for a smaller one, bit 1 for a larger one, an
// infinity or a NaN (magnitudes compared as integers, the sign shifted out).
__device__ __forceinline__ unsigned window_class(const float4 &v)
{
    const unsigned lo = 2u * __float_as_uint(xr::kWinLo), hi = 2u * __float_as_uint(xr::kWinHi);
    const unsigned a = 2u * __float_as_uint(v.x), b = 2u * __float_as_uint(v.y),
                   c = 2u * __float_as_uint(v.z), d = 2u * __float_as_uint(v.w);
    // 0 - 1 is the largest unsigned value
    return (unsigned)(min(min(a - 1u, b - 1u), min(c - 1u, d - 1u)) < lo - 1u) |
           ((unsigned)(max(max(a, b), max(c, d)) > hi) << 1);
}

// The same of every x and y tap of a warp's four rows (rows r0..r0+3 of a tile
// of tile_x; halo: the halo plane), shared among the lanes: 14 rows of the
// tile's 32 columns, and the 8 columns either side of the warp's own rows.
__device__ __forceinline__ unsigned halo_class(const float *halo, int r0, int tile_x)
{
    const int lane = threadIdx.x & 31, last = tile_x + 2 * kRadius - 1;
    unsigned cls = 0;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const int e = min(lane + 32 * i, 111);
        cls |= window_class(lds4(halo + min(r0 + (e >> 3), last) * kBoxY + kHaloY + 4 * (e & 7)));
    }
    const int row = min(r0 + kRadius + ((lane & 15) >> 2), last), c = lane & 3;
    return cls | window_class(lds4(halo + row * kBoxY + (c < 2 ? 4 * c : kTileY + 4 * c)));
}

// First derivatives only, for the gradmax kernels.
__device__ __forceinline__ void quad_grad_ref(const Taps &T, const Coefs &k, float Ux[4],
                                              float Uy[4], float Uz[4])
{
    const float *pc = T.pc;
    const float2 zero = make_float2(0.0f, 0.0f);
    float Y[20];
#pragma unroll
    for (int b = 0; b < 5; ++b) {
        float4 v = lds4(pc - 8 + 4 * b);
        Y[4 * b] = v.x; Y[4 * b + 1] = v.y; Y[4 * b + 2] = v.z; Y[4 * b + 3] = v.w;
    }
#pragma unroll
    for (int h = 0; h < 2; ++h) {
        const int j0 = 2 * h, j1 = 2 * h + 1;
        float2 g = zero;
#pragma unroll
        for (int m = 0; m < kRadius; ++m) {
            const float2 d = sub2(f2(Y[8 + j0 + m + 1], Y[8 + j1 + m + 1]),
                                  f2(Y[8 + j0 - m - 1], Y[8 + j1 - m - 1]));
            g = __fadd2_rn(g, div2(__fmul2_rn(k.rc[m], d), k.rh[1]));
        }
        Uy[j0] = g.x; Uy[j1] = g.y;
    }
    float2 gx[2] = {zero, zero}, gz[2] = {zero, zero};
#pragma unroll
    for (int m = 0; m < kRadius; ++m) {
        const float4 a = lds4(pc + (m + 1) * kBoxY);
        const float4 b = lds4(pc - (m + 1) * kBoxY);
        const float4 za = ztap(T, kRadius + m + 1);
        const float4 zb = ztap(T, kRadius - m - 1);
        const float2 a2[2] = {f2(a.x, a.y), f2(a.z, a.w)}, b2[2] = {f2(b.x, b.y), f2(b.z, b.w)};
        const float2 za2[2] = {f2(za.x, za.y), f2(za.z, za.w)},
                     zb2[2] = {f2(zb.x, zb.y), f2(zb.z, zb.w)};
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            gx[h] = __fadd2_rn(gx[h], div2(__fmul2_rn(k.rc[m], sub2(a2[h], b2[h])), k.rh[0]));
            gz[h] = __fadd2_rn(gz[h], div2(__fmul2_rn(k.rc[m], sub2(za2[h], zb2[h])), k.rh[2]));
        }
    }
    Ux[0] = gx[0].x; Ux[1] = gx[0].y; Ux[2] = gx[1].x; Ux[3] = gx[1].y;
    Uz[0] = gz[0].x; Uz[1] = gz[0].y; Uz[2] = gz[1].x; Uz[3] = gz[1].y;
}

// ---------------------------------------------------------------------------
// Plane pipeline.  The taps of a quad come from two rings.  The z taps need
// eleven planes, but of each only the tile's own cells: 4 KB a plane at 32
// rows.  The x and y taps need the 5-row, 8-column halo, but of the current
// plane only: 8 KB.  Iteration t (z = z0 + t) therefore waits for one group
// of loads: own-cell plane t + 10 (iteration 0: planes 0..10; plane i holds
// z = z0 - 5 + i, in slot i % (10 + G)) and halo plane t (slot t % G), both
// completing on full[t % G].  Eleven halo planes of 8 KB instead would leave
// no room for the step kernels' per-cell streams.
//
// A warp that has finished iteration t adds one to cnt[t % G]; the last one to
// do so refills what the iteration freed with group t + G (its
// own-cell plane goes to the slot of plane t, its halo plane to that of halo
// plane t).  No CTA barrier, no producer warp, and the load starts as soon as
// its slots are free.
// ---------------------------------------------------------------------------
template <int G> struct Pipe {
    float *zr, *cr;
    uint64_t *full;
    unsigned *cnt;
    int *issued;     // groups issued so far
    int zslot, cslot;
    unsigned zbytes, cbytes;
    int ngroups;     // iterations of this column
    int y0, x0, z0;
    int ncw;         // warps
    unsigned long long wait_ns;   // limit of every wait
    int hold;        // test hook: own-cell plane never loaded (-1: none)
};

template <int G>
__device__ __forceinline__ void pipe_issue(const Pipe<G> &P, const TileMaps *tm, int g)
{
    const int s = g % G;
    uint64_t *bar = &P.full[s];
    *P.issued = g + 1;
    mbar_arrive_expect_tx(bar, P.cbytes + P.zbytes * (g == 0 ? 2 * kRadius + 1 : 1));
    for (int i = g == 0 ? 0 : g + 2 * kRadius; i <= g + 2 * kRadius; ++i)
        if (i != P.hold)   // test hook: the wait for this group runs out
            tma_load_3d(P.zr + (i % ring_z(G)) * P.zslot, &tm->z, P.y0, P.x0, P.z0 - kRadius + i, bar);
    tma_load_3d(P.cr + s * P.cslot, &tm->c, P.y0 - kHaloY, P.x0 - kRadius, P.z0 + g, bar);
}

template <int G>
__device__ __forceinline__ bool pipe_wait(const Pipe<G> &P, int g)
{
    return mbar_wait_bounded(&P.full[g % G], (unsigned)((g / G) & 1), P.wait_ns);
}

// The end of a warp's iteration t (see above).
template <int G>
__device__ __forceinline__ void pipe_release(const Pipe<G> &P, const TileMaps *tm, int t)
{
    __syncwarp();
    if ((threadIdx.x & 31) == 0 && t + G < P.ngroups) {
        unsigned old;
        unsigned *c = &P.cnt[t % G];
        asm volatile("atom.acq_rel.cta.shared::cta.add.u32 %0, [%1], 1;"
                     : "=r"(old) : "r"(smem_u32(c)) : "memory");
        if (old == (unsigned)P.ncw - 1) {
            *c = 0;   // next used after the group issued here has landed
            fence_proxy_async();
            pipe_issue(P, tm, t + G);
        }
    }
}

// Thread 0, before a CTA barrier: barriers and counters, then the first groups.
template <int G>
__device__ void pipe_init(const Pipe<G> &P)
{
    for (int s = 0; s < G; ++s) {
        mbar_init(&P.full[s], 1);
        P.cnt[s] = 0;
    }
    fence_barrier_init();
    // a CTA that takes another tile reuses shared memory its threads read
    // and wrote (generic proxy) as TMA destination (async proxy)
    fence_proxy_async();
}

template <int G>
__device__ void pipe_start(const Pipe<G> &P, const TileMaps *tm)
{
    for (int g = 0; g < G && g < P.ngroups; ++g) pipe_issue(P, tm, g);
}

// The end of a column: true if no wait ran out (the same in every thread).
// Otherwise the loads still in flight are waited for (bounded), so that none
// lands in shared memory after the CTA has exited.
template <int G>
__device__ bool pipe_finish(const Pipe<G> &P, bool ok, unsigned *err)
{
    if (__syncthreads_and(ok)) return true;
    if (threadIdx.x == 0) {
        atomicOr(err, kErrWaitTimeout);
        for (int g = max(0, *P.issued - G); g < *P.issued; ++g) (void)pipe_wait(P, g);
    }
    return false;
}

template <int G>
__device__ __forceinline__ void pipe_setup(Pipe<G> &P, unsigned char *smem, const SmemLayout &L,
                                           int tile_x, int y0, int x0, int z0, int nzc)
{
    P.zr = reinterpret_cast<float *>(smem);
    P.cr = reinterpret_cast<float *>(smem + L.c_off);
    P.full = reinterpret_cast<uint64_t *>(smem + L.bar_off);
    P.cnt = reinterpret_cast<unsigned *>(smem + L.cnt_off);
    P.issued = reinterpret_cast<int *>(P.cnt + G);
    P.zslot = L.zslot;
    P.cslot = L.cslot;
    P.zbytes = (unsigned)(tile_x * kTileY * 4);
    P.cbytes = (unsigned)((tile_x + 2 * kRadius) * kBoxY * 4);
    P.ngroups = nzc;
    P.y0 = y0;
    P.x0 = x0;
    P.z0 = z0;
    P.ncw = blockDim.x >> 5;   // every warp of the CTA releases every iteration
    P.wait_ns = 2000000000ull;
    P.hold = -1;
}

// The launch's wait limit (0: 2 s) and the plane-withholding test hook (the
// first CTA of a grid launch only).
template <int G>
__device__ __forceinline__ void pipe_hooks(Pipe<G> &P, unsigned long long wait_ns, int hold_plane)
{
    if (wait_ns) P.wait_ns = wait_ns;
    if (hold_plane > 0 && (blockIdx.x | blockIdx.y | blockIdx.z) == 0) P.hold = hold_plane - 1;
}

// Before a CTA reuses its barriers for another tile (thread 0, after a CTA
// barrier; every load of the previous tile has been waited for).
template <int G>
__device__ void pipe_inval(const Pipe<G> &P)
{
    for (int s = 0; s < G; ++s)
        asm volatile("mbarrier.inval.shared::cta.b64 [%0];" ::"r"(smem_u32(&P.full[s])) : "memory");
}

// The ring positions of iteration t, kept incrementally.
template <int G>
__device__ __forceinline__ Taps taps_start(const Pipe<G> &P, int r, int q)
{
    Taps T;
    T.pc = P.cr + (r + kRadius) * kBoxY + kHaloY + 4 * q;
    T.za = P.zr + r * kTileY + 4 * q;
    T.wrap = ring_z(G);
    T.zslot = P.zslot;
    T.zlen = ring_z(G) * P.zslot;
    return T;
}

template <int G>
__device__ __forceinline__ void taps_next(Taps &T, const Pipe<G> &P, int t)   // from t to t + 1
{
    T.za += T.zslot;
    if (--T.wrap == 0) {
        T.za -= T.zlen;
        T.wrap = ring_z(G);
    }
    T.pc += t % G == G - 1 ? -(G - 1) * P.cslot : P.cslot;
}

// ---------------------------------------------------------------------------
// max|grad u| over one tile column [z0, z1), one per CTA, a warp's maximum in
// mx.  Returns false (in every thread) when a wait timed out.
// ---------------------------------------------------------------------------
template <int AR>
__device__ __forceinline__ bool gradmax_tile(const TileMaps *tm, const PlaneParams &p,
                                             const Coefs &k, int tile_x, int y0, int x0, int z0,
                                             int z1, unsigned char *smem, float &mx)
{
    const int tid = threadIdx.x;
    const int q = tid & (kQuadsY - 1), r = tid / kQuadsY;
    const int nzc = z1 - z0;
    const SmemLayout L = smem_layout(tile_x, 0, 0, 0, kGradmaxGroups);
    Pipe<kGradmaxGroups> P;
    pipe_setup(P, smem, L, tile_x, y0, x0, z0, nzc);
    pipe_hooks(P, p.wait_ns, p.hold_plane);
    if (tid == 0) {
        pipe_init(P);
        pipe_start(P, tm);
    }
    __syncthreads();
    const int x = x0 + r, yq = y0 + 4 * q;
    const bool row_ok = (r < tile_x) && (x < p.nx - kRadius);
    bool cell_ok[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) cell_ok[j] = row_ok && (yq + j >= kRadius) && (yq + j < p.ny - kRadius);
    Taps T = taps_start(P, r, q);
    mx = 0.0f;
    bool ok = true;
    for (int t = 0; t < nzc; taps_next(T, P, t), ++t) {
        ok = __all_sync(0xffffffffu, pipe_wait(P, t));
        if (!ok) break;
        if (row_ok) {
            float Ux[4], Uy[4], Uz[4], Uxx[4], Uyy[4], Uzz[4], u0[4];
            if (AR == kArithRef) quad_grad_ref(T, k, Ux, Uy, Uz);
            else quad_derivs<false>(T, k, Ux, Uy, Uz, Uxx, Uyy, Uzz, u0);
#pragma unroll
            for (int j = 0; j < 4; ++j)
                if (cell_ok[j])
                    mx = fmaxf(mx, fmaxf(fabsf(Ux[j]), fmaxf(fabsf(Uy[j]), fabsf(Uz[j]))));
        }
        pipe_release(P, tm, t);
    }
    ok = pipe_finish(P, ok, p.err);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
    return ok;
}

__device__ __forceinline__ void gradmax_publish(const PlaneParams &p, float mx)
{
    if ((threadIdx.x & 31) == 0 && mx > 0.0f)
        atomicMax(reinterpret_cast<unsigned *>(p.gmax + p.step), __float_as_uint(mx));
}

template <int AR>
__global__ void __launch_bounds__(kThreads, 2)
    qp3d_gradmax_kernel(const __grid_constant__ TileMaps tm, const PlaneParams p)
{
    extern __shared__ __align__(128) unsigned char smem[];
    pdl_trigger();
    pdl_wait();
    const int z0 = kRadius + blockIdx.z * p.chunk_z;
    const int z1 = min(z0 + p.chunk_z, p.nz - kRadius);
    if (z0 >= z1) return;
    float mx;
    gradmax_tile<AR>(&tm, p, p.k, p.tile_x, blockIdx.x * kTileY,
                     kRadius + blockIdx.y * p.tile_x, z0, z1, smem, mx);
    gradmax_publish(p, mx);
}

// ---------------------------------------------------------------------------
// gradmax for a caller that supplies no buffer: the maximum, a count of the
// CTAs that are done and the error word live in one small scratch that every
// launch finds zero.  The last CTA delivers the result (NaN when a wait ran
// out) and the error flags, and leaves the scratch zero again.
// ---------------------------------------------------------------------------
__device__ __forceinline__ void gradmax_deliver(GradmaxScratch *sc, float *out,
                                                unsigned *host_flags)
{
    __syncthreads();
    if (threadIdx.x != 0) return;
    __threadfence();
    if (atomicAdd(&sc->done, 1u) != gridDim.x * gridDim.y * gridDim.z - 1) return;
    __threadfence();
    const unsigned flags = atomicExch(&sc->err, 0u), bits = atomicExch(&sc->max_bits, 0u);
    atomicExch(&sc->done, 0u);
    out[0] = flags ? __int_as_float(0x7fc00000) : __uint_as_float(bits);
    *host_flags = flags;
}

__global__ void __launch_bounds__(kQuadsY * kGradmaxTileX, 4)
    qp3d_gradmax_single_kernel(const __grid_constant__ TileMaps tm, const PlaneParams p,
                               GradmaxScratch *sc, float *out, unsigned *host_flags)
{
    extern __shared__ __align__(128) unsigned char smem[];
    // tiles of a plane in the grid's first dimension, which has no limit of 65535
    const int nyt = (p.ny - kRadius - 1) / kTileY + 1;
    const int yt = blockIdx.x % nyt, xt = blockIdx.x / nyt;
    const int z0 = kRadius + blockIdx.z * p.chunk_z;
    const int z1 = min(z0 + p.chunk_z, p.nz - kRadius);
    if (z0 < z1) {
        float mx;
        gradmax_tile<kArithFast>(&tm, p, p.k, p.tile_x, yt * kTileY,
                                 kRadius + xt * p.tile_x, z0, z1, smem, mx);
        if ((threadIdx.x & 31) == 0 && mx > 0.0f) atomicMax(&sc->max_bits, __float_as_uint(mx));
    }
    gradmax_deliver(sc, out, host_flags);
}

// The same without staging: a thread marches along z with one quad, its own
// column of eleven planes in registers (the loop is unrolled by eleven, so that
// the queue never moves), and takes the x and y taps through L1: fifteen
// 16-byte loads a quad and plane instead of the staged form's 25 from shared
// memory, and no barriers or copies to wait for on a small grid.  240x240x190:
// 49 us a call, 60 staged; held to 3, 5 or 6 CTAs an SM 59, 62 and 75 (fewer warps,
// or spills).
constexpr int kDirectThreads = 128;   // 8 quads by 16 rows
__global__ void __launch_bounds__(kDirectThreads, 4)
    qp3d_gradmax_direct_kernel(const float *u, int nx, int ny, int nz, int ldy, int chunk_z,
                               const __grid_constant__ Coefs k, GradmaxScratch *sc, float *out,
                               unsigned *host_flags)
{
    constexpr int N = 2 * kRadius + 1;
    const int q = threadIdx.x & 7, x = kRadius + blockIdx.y * (kDirectThreads / 8) + (threadIdx.x >> 3);
    const int y = blockIdx.x * kTileY + 4 * q;
    const int z0 = kRadius + blockIdx.z * chunk_z, z1 = min(z0 + chunk_z, nz - kRadius);
    float mx = 0.0f;
    unsigned okb = 0;   // bits of the quad's updated cells
#pragma unroll
    for (int j = 0; j < 4; ++j)
        if (y + j >= kRadius && y + j < ny - kRadius) okb |= 1u << j;
    if (okb && x < nx - kRadius) {
        const size_t plane = (size_t)nx * ldy;
        const float *c = u + (size_t)z0 * plane + (size_t)x * ldy + y;   // the current plane's quad
        auto ld = [](const float *p) { return __ldg(reinterpret_cast<const float4 *>(p)); };
        const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
        float4 zq[N];   // slot (z - z0 + 5 + d) % 11 holds plane z + d
#pragma unroll
        for (int i = 0; i < 2 * kRadius; ++i)
            zq[i] = ld(c + (ptrdiff_t)(i - kRadius) * (ptrdiff_t)plane);
        for (int t0 = z0; t0 < z1; t0 += N) {
#pragma unroll
            for (int t = 0; t < N; ++t) {
                if (t0 + t >= z1) break;
                zq[(t + 2 * kRadius) % N] = ld(c + kRadius * plane);
                float Y[20];
#pragma unroll
                for (int b = 0; b < 5; ++b) {
                    const int yb = y - 8 + 4 * b;
                    const float4 v = b == 2 ? zq[(t + kRadius) % N]
                                   : yb >= 0 && yb < ldy ? ld(c - 8 + 4 * b) : zero;
                    Y[4 * b] = v.x; Y[4 * b + 1] = v.y; Y[4 * b + 2] = v.z; Y[4 * b + 3] = v.w;
                }
                float2 gx[2], gy[2], gz[2];
#pragma unroll
                for (int m = 0; m < kRadius; ++m) {
                    const float4 xp = ld(c + (m + 1) * ldy), xm = ld(c - (m + 1) * ldy);
#pragma unroll
                    for (int h = 0; h < 2; ++h) {
                        const int j0 = 8 + 2 * h;
                        const float2 dx = sub2(half2of(xp, h), half2of(xm, h));
                        const float2 dy = sub2(f2(Y[j0 + m + 1], Y[j0 + m + 2]),
                                               f2(Y[j0 - m - 1], Y[j0 - m]));
                        const float2 dz = sub2(half2of(zq[(t + kRadius + m + 1) % N], h),
                                               half2of(zq[(t + kRadius - m - 1) % N], h));
                        gx[h] = m == 0 ? __fmul2_rn(k.cx2[0], dx) : __ffma2_rn(k.cx2[m], dx, gx[h]);
                        gy[h] = m == 0 ? __fmul2_rn(k.cy2[0], dy) : __ffma2_rn(k.cy2[m], dy, gy[h]);
                        gz[h] = m == 0 ? __fmul2_rn(k.cz2[0], dz) : __ffma2_rn(k.cz2[m], dz, gz[h]);
                    }
                }
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    if ((okb >> (2 * h)) & 1u)
                        mx = fmaxf(mx, fmaxf(fabsf(gx[h].x), fmaxf(fabsf(gy[h].x), fabsf(gz[h].x))));
                    if ((okb >> (2 * h + 1)) & 1u)
                        mx = fmaxf(mx, fmaxf(fabsf(gx[h].y), fmaxf(fabsf(gy[h].y), fabsf(gz[h].y))));
                }
                c += plane;
            }
        }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
    if ((threadIdx.x & 31) == 0 && mx > 0.0f) atomicMax(&sc->max_bits, __float_as_uint(mx));
    gradmax_deliver(sc, out, host_flags);
}

// ---------------------------------------------------------------------------
// PML update of a quad in the fast arithmetic (GPU_kernel.cu:566-637 restated
// with per-layer coefficients a1 = (d*dt+1)^2-3, a2 = 2*d*dt-1, a3 = 1-dt*d),
// for faces normal to axis AX (0 x, 1 y, 2 z), two cells at a time with the
// packed FP32x2 instructions.  na1 = -a1, and dd carries the sign of the odd
// faces (R, Bk, Bo), so that every product and sum rounds as the scalar
// expression does.  One body per axis: choosing the normal and tangential
// derivatives of every cell by selects took about a third of the update's
// instructions.
// ---------------------------------------------------------------------------
struct PmlOwn {   // what a PML quad reads of its split-field state
    float4 w11, w12, w31, w32, p1, p2, w21;
};
struct PmlNew {
    float2 w13[2], w21[2], w33[2], p3[2];
};

template <int AX>
__device__ __forceinline__ float2 pml_pair(float2 na1, float2 a2, float2 a3, float2 dd, float2 KS,
                                           float2 e1, float2 Un, float2 Uxx, float2 Uyy,
                                           float2 Uzz, float2 dt, const PmlOwn &o, int h,
                                           PmlNew &n)
{
    const float2 e2KS = __fmul2_rn(e1, KS);
    const float2 A = AX == 2 ? KS : e2KS, Bt = AX == 2 ? e2KS : KS;
    const float2 Unn = AX == 0 ? Uxx : AX == 1 ? Uyy : Uzz;
    const float2 Tt = AX == 2 ? __fadd2_rn(Uxx, Uyy) : __ffma2_rn(e1, AX == 0 ? Uyy : Uxx, Uzz);
    n.w13[h] = __ffma2_rn(A, Unn, __ffma2_rn(na1, half2of(o.w12, h),
                                             __fmul2_rn(a2, half2of(o.w11, h))));
    n.p3[h] = __ffma2_rn(__fmul2_rn(A, dd), Un, __ffma2_rn(na1, half2of(o.p2, h),
                                                           __fmul2_rn(a2, half2of(o.p1, h))));
    n.w21[h] = __ffma2_rn(dt, n.p3[h], __fmul2_rn(a3, half2of(o.w21, h)));
    const float2 w31 = half2of(o.w31, h);
    const float2 X3 = __ffma2_rn(make_float2(2.0f, 2.0f), half2of(o.w32, h),
                                 make_float2(-w31.x, -w31.y));
    n.w33[h] = __ffma2_rn(Bt, Tt, X3);
    return __fadd2_rn(__fadd2_rn(n.w13[h], n.w21[h]), n.w33[h]);
}

// Face code and layer index of a cell from its x/y/z face parts (-1: none),
// in the reference's priority order.
__device__ __forceinline__ void cell_face(int fx, int lix, int fy, int liy, int fz, int liz,
                                          int &f, int &li)
{
    f = fx >= 0 ? fx : (fy >= 0 ? fy : fz);
    li = fx >= 0 ? lix : (fy >= 0 ? liy : liz);
}

// ---------------------------------------------------------------------------
// step kernel.
//   SPEC = false ("exact"): the threshold comes from gmax[step], already
//     known (gradmax kernel, or a speculative pass of the same step whose
//     resolution found that it has to be re-run).
//   SPEC = true: the max of the step is not known yet.  It is predicted from
//     the two previous steps with a window [M_lo, M_hi]; a cell whose m2 lies
//     in (T2(M_lo), T2(M_hi)] has an uncertain decision: the kernel computes
//     it as "above", lists it in its column's segment with its m2 and what
//     gives it its S = 1 result, and reduces the true max of the step into
//     gmax[step] on the way.  The resolution kernel then gives the S = 1
//     result to the listed cells that turn out to be below the threshold, or
//     runs the exact step again when the max fell outside the window or a
//     segment was too short.  The step never overwrites its inputs, so both
//     are possible.  Both modes write bit-identical results.
// ---------------------------------------------------------------------------
// w = (M_lo, M_hi, M_pred) of step k, from the maxima of the two steps before
// and the recent prediction errors.
__device__ void spec_window(const PlaneParams &p, int k, const float *spec_err, float w[3])
{
    const float m1 = k >= 1 ? p.gmax[k - 1] : 0.0f;
    const float m0 = k >= 2 ? p.gmax[k - 2] : 0.0f;
    float r = (m0 > 0.0f) ? __fdiv_rn(m1, m0) : 1.0f;
    r = fminf(fmaxf(r, 0.5f), 2.0f);
    // half the last trend: late in a shot the max moves by a few tenths of a
    // percent per step with changing sign, which a full extrapolation doubles
    const float pred = __fmul_rn(m1, fmaf(0.5f, __fsub_rn(r, 1.0f), 1.0f));
    // cover both "the max keeps its trend" and "the max stays where it was",
    // widened by 1.5x the largest of the recent prediction errors
    float e = 0.0f;
#pragma unroll
    for (int i = 0; i < kSpecHist; ++i) e = fmaxf(e, spec_err[i]);
    const float d = fminf(0.25f, fmaxf(p.delta_min, __fmul_rn(1.5f, e)));
    w[0] = __fmul_rn(fminf(pred, m1), __fsub_rn(1.0f, d));
    w[1] = __fmul_rn(fmaxf(pred, m1), __fadd_rn(1.0f, d));
    w[2] = pred;
    if (p.spec_bias != 0.0f) {   // test hook: a window that misses on purpose
        w[0] = __fmul_rn(w[0], __fadd_rn(1.0f, p.spec_bias));
        w[1] = __fmul_rn(w[1], __fadd_rn(1.0f, p.spec_bias));
    }
}

// 1/x for normal positive x, within about 1 ulp: Newton-Raphson steps
// r <- r + r (1 - x r) from an initial guess that negates the exponent of x in
// its integer representation (the integer-subtraction trick known from the
// fast inverse square root).  Three steps take the guess's ~12% error below
// float rounding.  About a third of the instructions of an IEEE division,
// which dominated the scalar operator once most cells are above the
// threshold; the mirror oracle performs the same operations:
//   r = bits(0x7EF311C3 - bits(x)); 3 x { e = fma(-x, r, 1); r = fma(r, e, r) }
// Two cells at a time with the packed FP32x2 instructions (round-to-nearest
// per lane: each lane performs the scalar operations above).
__device__ __forceinline__ float2 rcp_nr2(float2 x)
{
    float2 r = make_float2(__uint_as_float(0x7EF311C3u - __float_as_uint(x.x)),
                           __uint_as_float(0x7EF311C3u - __float_as_uint(x.y)));
    const float2 nx = make_float2(-x.x, -x.y), one = make_float2(1.0f, 1.0f);
#pragma unroll
    for (int it = 0; it < 3; ++it) {
        const float2 e = __ffma2_rn(nx, r, one);
        r = __ffma2_rn(r, e, r);
    }
    return r;
}

// S of two cells (GPU_kernel.cu:100-111), given they are above the threshold.
// With a = (nx^2 + ny^2) = h2/m2, nz^2 = 1 - a = v2/m2 (v2 = Uz^2),
// S = 1/2 + 1/2 sqrt(1 - 8(eps-delta) a (1-a) / (1 + 2 eps a)^2)
//   = 1/2 + 1/2 sqrt(1 - 8(eps-delta) (h2 r) (v2 r)),  r = 1 / (m2 + 2 eps h2):
// one reciprocal per cell, and both factors h2 r, v2 r lie in [0, 1].
__device__ __forceinline__ float2 aniso_s2(float2 h2, float2 m2, float2 v2, float2 e2x, float2 r8)
{
    const float2 one = make_float2(1.0f, 1.0f), half = make_float2(0.5f, 0.5f);
    const float2 r = rcp_nr2(__ffma2_rn(e2x, h2, m2));
    const float2 qq = __fmul2_rn(__fmul2_rn(r8, __fmul2_rn(h2, r)), __fmul2_rn(v2, r));
    const float2 t = __fadd2_rn(one, make_float2(-qq.x, -qq.y));
    return __ffma2_rn(half, make_float2(__fsqrt_rn(t.x), __fsqrt_rn(t.y)), half);
}

// Per-cell parameters of a quad from half-precision vp, eps, delta, with the
// operations of qp3d_params_dense_kernel: vp, 2 eps, 8 (eps - delta).
__device__ __forceinline__ void quad_params_half(uint2 hv, uint2 he, uint2 hd, float4 &V,
                                                 float4 &E2, float4 &R8)
{
    const float2 v0 = __half22float2(*reinterpret_cast<const __half2 *>(&hv.x));
    const float2 v1 = __half22float2(*reinterpret_cast<const __half2 *>(&hv.y));
    const float2 e0 = __half22float2(*reinterpret_cast<const __half2 *>(&he.x));
    const float2 e1 = __half22float2(*reinterpret_cast<const __half2 *>(&he.y));
    const float2 d0 = __half22float2(*reinterpret_cast<const __half2 *>(&hd.x));
    const float2 d1 = __half22float2(*reinterpret_cast<const __half2 *>(&hd.y));
    const float ep[4] = {e0.x, e0.y, e1.x, e1.y}, de[4] = {d0.x, d0.y, d1.x, d1.y};
    float e[4], r[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        e[j] = __fmul_rn(2.0f, ep[j]);
        r[j] = __fmul_rn(8.0f, __fsub_rn(ep[j], de[j]));
    }
    V = make_float4(v0.x, v0.y, v1.x, v1.y);
    E2 = make_float4(e[0], e[1], e[2], e[3]);
    R8 = make_float4(r[0], r[1], r[2], r[3]);
}

// (vp dt)^2 of the fast arithmetic
__device__ __forceinline__ float k_of_vp(float vp, float dt)
{
    const float vdt = __fmul_rn(vp, dt);
    return __fmul_rn(vdt, vdt);
}

// The fast arithmetic's layer coefficients from the stored (a1h, a1l, d*dt, dd):
// a1 = RN(a1h + a1l) = a1h, a2 = 2*d*dt - 1, a3 = 1 - d*dt.
__device__ __forceinline__ float4 fast_layer(float4 t)
{
    return make_float4(t.x, __fmaf_rn(2.0f, t.z, -1.0f), __fsub_rn(1.0f, t.z), t.w);
}

// The same with -a1 in place of a1, as the packed PML update takes it.
__device__ __forceinline__ float4 step_layer(float4 t)
{
    const float4 l = fast_layer(t);
    return make_float4(-l.x, l.y, l.z, l.w);
}

// The split-field update of one PML cell of face code f, layer li; v: its
// pml_inputs, ks as in step_tile.
// (Not inlined, as scalar_s_call: four copies each in two loop bodies did not
// stay in the instruction cache; 2-5 % of a step in the reference arithmetic.)
template <int AR>
__device__ __noinline__ xr::PmlOut pml_cell(int f, float4 layer, float ks, float e1, float vp,
                                               float4 v, float dt, float w11, float w12, float w21,
                                               float w31, float w32, float p1, float p2)
{
    const bool isz = f >= 4;
    if (AR == kArithRef) {
        xr::PmlLayer Lr;
        Lr.a1h = layer.x; Lr.a1l = layer.y;
        Lr.a2 = __fmaf_rn(2.0f, layer.z, -1.0f);
        Lr.a3 = __fsub_rn(1.0f, layer.z);
        Lr.dd = layer.w;
        return xr::pml_update(isz, (f & 1) != 0, ks, e1, __fmul_rn(vp, dt), v.x, v.y, v.z, dt, Lr,
                              w11, w12, w21, w31, w32, p1, p2);
    }
    const float4 lc = step_layer(layer);
    const float e2KS = __fmul_rn(e1, ks);
    const float A = isz ? ks : e2KS, Bt = isz ? e2KS : ks;
    xr::PmlOut o;
    o.w13 = fmaf(A, v.x, fmaf(lc.x, w12, __fmul_rn(lc.y, w11)));
    o.p3 = fmaf(__fmul_rn(A, (f & 1) ? -lc.w : lc.w), v.y, fmaf(lc.x, p2, __fmul_rn(lc.y, p1)));
    o.w21 = fmaf(dt, o.p3, __fmul_rn(lc.z, w21));
    o.w33 = fmaf(Bt, v.z, fmaf(2.0f, w32, -w31));
    o.u3 = __fadd_rn(__fadd_rn(o.w13, o.w21), o.w33);
    return o;
}

// Where the cells of one column that wait for the exact max are listed
// ("deferred" cells): a segment of the shot's list, in no particular order,
// with its length.
struct DeferSeg {
    size_t base;        // first entry of the segment
    unsigned cap;       // its entries; more deferred cells make the step re-run
    unsigned *count;
};

// The interior update, S of the cell as kS above: the reference's roundings, or
// two fused multiply-adds.
template <int AR>
__device__ __forceinline__ float interior_cell(float u0, float u1, float Uxx, float Uyy, float Uzz,
                                               float e1, float ks, float vp, float dt2)
{
    if (AR == kArithRef) return xr::interior_update(u0, u1, Uxx, Uyy, Uzz, e1, ks, vp, dt2);
    const float Lp = fmaf(e1, __fadd_rn(Uxx, Uyy), Uzz);
    return fmaf(ks, Lp, fmaf(2.0f, u0, -u1));
}

// Places in the segment for the deferred cells of a warp's quads (nib: a bit
// per cell): the first place of this thread's.  *cnt: the segment's length so
// far, in shared memory.
__device__ __forceinline__ unsigned defer_places(unsigned *cnt, unsigned nib)
{
    const unsigned lane = threadIdx.x & 31;
    const unsigned c = __popc(nib);
    unsigned incl = c;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const unsigned v = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= (unsigned)o) incl += v;
    }
    unsigned first = 0;
    if (lane == 31) first = atomicAdd(cnt, incl);
    return __shfl_sync(0xffffffffu, first, 31) + incl - c;
}

// The derivatives the PML update of a face code f takes: along the normal
// (second, first) and the tangential combination.
template <int AR>
__device__ __forceinline__ float4 pml_inputs(int f, float e1, float Ux, float Uy, float Uz,
                                             float Uxx, float Uyy, float Uzz)
{
    const bool isx = f < 2, isz = f >= 4;
    const float Ut = isx ? Uyy : Uxx;
    float Tt;
    if (isz) Tt = __fadd_rn(Uxx, Uyy);
    else Tt = AR == kArithRef ? __fadd_rn(Uzz, __fmul_rn(e1, Ut)) : fmaf(e1, Ut, Uzz);
    return make_float4(isx ? Uxx : (isz ? Uzz : Uyy), isx ? Ux : (isz ? Uz : Uy), Tt, 0.0f);
}

// Largest and smallest of four values, NaN if any is: a comparison with it is
// then false, as the comparison with that value is.
__device__ __forceinline__ float max4(const float v[4])
{
    float r;
    asm("max.NaN.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(v[0]), "f"(v[1]), "f"(v[2]));
    asm("max.NaN.f32 %0, %1, %2;" : "=f"(r) : "f"(r), "f"(v[3]));
    return r;
}
__device__ __forceinline__ float min4(const float v[4])
{
    float r;
    asm("min.NaN.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(v[0]), "f"(v[1]), "f"(v[2]));
    asm("min.NaN.f32 %0, %1, %2;" : "=f"(r) : "f"(r), "f"(v[3]));
    return r;
}

// The PML update of a quad, its interior results in out: the cells of pmlb get
// the split-field ones, and n every new state (0, and the old w21, for cells
// that are not of the shell).
__device__ __forceinline__ void pml_quad_ref(
    const PlaneParams &p, const float4 *tab, const float kS[4], const float e1[4], float4 Vv,
    const float Ux[4], const float Uy[4], const float Uz[4], const float Uxx[4],
    const float Uyy[4], const float Uzz[4], const PmlOwn &o, unsigned pmlb, int fx, int lix,
    int yq, int fz, int liz, float out[4], PmlNew &n)
{
    const int pml = p.pml, ny = p.ny;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        float *w13 = j & 1 ? &n.w13[j >> 1].y : &n.w13[j >> 1].x;
        float *w21 = j & 1 ? &n.w21[j >> 1].y : &n.w21[j >> 1].x;
        float *w33 = j & 1 ? &n.w33[j >> 1].y : &n.w33[j >> 1].x;
        float *p3 = j & 1 ? &n.p3[j >> 1].y : &n.p3[j >> 1].x;
        *w13 = *w33 = *p3 = 0.0f;
        *w21 = f4(o.w21, j);
        if (!((pmlb >> j) & 1u)) continue;
        int f, li;
        const int y = yq + j;
        const int fy = y < pml ? 2 : (y >= ny - pml ? 3 : -1);
        cell_face(fx, lix, fy, y < pml ? pml - y : y - ny + pml, fz, liz, f, li);
        const xr::PmlOut v = pml_cell<kArithRef>(
            f, tab[(f >> 1) * pml + li], kS[j], e1[j], f4(Vv, j),
            pml_inputs<kArithRef>(f, e1[j], Ux[j], Uy[j], Uz[j], Uxx[j], Uyy[j], Uzz[j]), p.dt,
            f4(o.w11, j), f4(o.w12, j), f4(o.w21, j), f4(o.w31, j), f4(o.w32, j), f4(o.p1, j),
            f4(o.p2, j));
        out[j] = v.u3;
        *w13 = v.w13; *w21 = v.w21; *w33 = v.w33; *p3 = v.p3;
    }
}

__device__ __forceinline__ void pml_quad_fast(
    const PlaneParams &p, const float4 *tab, const float *ytab, const float kS[4],
    const float e1[4], const float Ux[4], const float Uy[4], const float Uz[4],
    const float Uxx[4], const float Uyy[4], const float Uzz[4], const PmlOwn &o, unsigned pmlb,
    unsigned fyb, int fx, int lix, int fz, int liz, float out[4], PmlNew &n)
{
    const float2 dt = make_float2(p.dt, p.dt);
    float2 v[2];
#define QP3D_PML_PAIRS(AX, NA1, A2, A3, DD, UN)                                                   _Pragma("unroll") for (int h = 0; h < 2; ++h) {                                                   const int j0 = 2 * h, j1 = 2 * h + 1;                                                         v[h] = pml_pair<AX>(NA1, A2, A3, DD, f2(kS[j0], kS[j1]), f2(e1[j0], e1[j1]),                                      f2(UN[j0], UN[j1]), f2(Uxx[j0], Uxx[j1]), f2(Uyy[j0], Uyy[j1]),                               f2(Uzz[j0], Uzz[j1]), dt, o, h, n);                                   }
    if (fx >= 0) {
        const float4 lc = tab[lix];
        const float dd = fx ? -lc.w : lc.w;
        QP3D_PML_PAIRS(0, f2(lc.x, lc.x), f2(lc.y, lc.y), f2(lc.z, lc.z), f2(dd, dd), Ux)
    } else if (fyb) {
        const float4 c1 = lds4(ytab), c2 = lds4(ytab + kTileY), c3 = lds4(ytab + 2 * kTileY),
                     c4 = lds4(ytab + 3 * kTileY);
        QP3D_PML_PAIRS(1, half2of(c1, h), half2of(c2, h), half2of(c3, h), half2of(c4, h), Uy)
        if (fyb != 15u && fz >= 0) {   // the quad's other cells are of the z face
            const PmlNew y = n;
            const float2 vy[2] = {v[0], v[1]};
            const float4 lc = tab[2 * p.pml + liz];
            const float dd = fz & 1 ? -lc.w : lc.w;
            QP3D_PML_PAIRS(2, f2(lc.x, lc.x), f2(lc.y, lc.y), f2(lc.z, lc.z), f2(dd, dd), Uz)
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                if (fyb >> (2 * h) & 1u) {
                    v[h].x = vy[h].x;
                    n.w13[h].x = y.w13[h].x; n.w21[h].x = y.w21[h].x;
                    n.w33[h].x = y.w33[h].x; n.p3[h].x = y.p3[h].x;
                }
                if (fyb >> (2 * h + 1) & 1u) {
                    v[h].y = vy[h].y;
                    n.w13[h].y = y.w13[h].y; n.w21[h].y = y.w21[h].y;
                    n.w33[h].y = y.w33[h].y; n.p3[h].y = y.p3[h].y;
                }
            }
        }
    } else {
        const float4 lc = tab[2 * p.pml + liz];
        const float dd = fz & 1 ? -lc.w : lc.w;
        QP3D_PML_PAIRS(2, f2(lc.x, lc.x), f2(lc.y, lc.y), f2(lc.z, lc.z), f2(dd, dd), Uz)
    }
#undef QP3D_PML_PAIRS
    if (pmlb == 15u) {
        out[0] = v[0].x; out[1] = v[0].y; out[2] = v[1].x; out[3] = v[1].y;
        return;
    }
#pragma unroll
    for (int h = 0; h < 2; ++h) {   // cells of the interior or of the never-updated band
        if (pmlb >> (2 * h) & 1u) {
            out[2 * h] = v[h].x;
        } else {
            n.w13[h].x = n.w33[h].x = n.p3[h].x = 0.0f;
            n.w21[h].x = half2of(o.w21, h).x;
        }
        if (pmlb >> (2 * h + 1) & 1u) {
            out[2 * h + 1] = v[h].y;
        } else {
            n.w13[h].y = n.w33[h].y = n.p3[h].y = 0.0f;
            n.w21[h].y = half2of(o.w21, h).y;
        }
    }
}

__device__ __noinline__ float scalar_s_call(float Ux, float Uy, float Uz, float m2, float e,
                                            float r)
{
    return xr::scalar_s(Ux, Uy, Uz, m2, e, r);
}

// One tile column [z0, z1) of the step.  The step kernels, single and batched,
// run one per CTA; the re-runs in the resolution kernels run many (REUSE:
// barriers invalidated at the end).  The return value is the same in every
// thread; false = a wait timed out.
// AR: kArithRef (the reference CPU operators' roundings, qp3d_exact.h) or
// kArithFast (folded coefficients, fused multiply-adds, one reciprocal in S).
// DEC: the step's threshold decisions are kept or replayed (p.dec_out,
// p.dec_in) where asked for.
template <bool SPEC, bool REUSE, bool HALF, int AR, bool DEC>
__device__ __forceinline__ bool step_tile(const TileMaps *tm, const PlaneParams &p,
                                          const Coefs &k, int tile_x, int y0, int x0, int z0,
                                          int z1, bool win_writer, const DeferSeg &seg,
                                          unsigned char *smem)
{
    const SmemLayout L = smem_layout(tile_x, p.pml, p.nsrc, step_streams(p.pml));
    float4 *tab = reinterpret_cast<float4 *>(smem + L.tab_off);
    float *ytab = reinterpret_cast<float *>(smem + L.ytab_off);
    SrcEntry *csrc = reinterpret_cast<SrcEntry *>(smem + L.src_off);
    float *misc = reinterpret_cast<float *>(smem + L.misc_off);
    unsigned *misc_u = reinterpret_cast<unsigned *>(smem + L.misc_off + 16);

    const int tid = threadIdx.x, lane = tid & 31;
    // A warp holds four rows of eight quads, or, in a last y tile of no more
    // than four or two quads, eight or sixteen rows: the warps left over only
    // pass the planes on.  (A last tile starts at ny - 6 or before: two quads.)  (Decision words and the reference
    // arithmetic's classes go by rows of eight.)  A step of 140^3 cells (last
    // tile 12 wide) 45.3 -> 42.5 us, 38x42x34 10.5 -> 10.1, 191x127x105 (31
    // wide) 35.7 -> 35.1, 240x240x190 (16) 107.5 -> 106.4.
    int lq = 3;
    if (AR == kArithFast && !DEC) {
        const int nq = (min(p.ny - y0, kTileY) + 3) >> 2;
        lq = nq > 4 ? 3 : (nq > 2 ? 2 : 1);
    }
    const int q = tid & ((1 << lq) - 1), r = tid >> lq, rt = min(r, tile_x - 1);
    const int nzc = z1 - z0;
    Pipe<kGroups> P;
    pipe_setup(P, smem, L, tile_x, y0, x0, z0, nzc);
    if (!REUSE) pipe_hooks(P, p.wait_ns, p.hold_plane);
    const int nx = p.nx, ny = p.ny, nz = p.nz, pml = p.pml;
    const int x = x0 + r, yq = y0 + 4 * q;
    const bool row_ok = (r < tile_x) && (x < nx - kRadius);
    // quads wholly in the row padding (y >= ny, the last y tile) neither load
    // nor store: their cells are not part of the volume
    const bool mem_ok = row_ok && (yq < ny);
    const bool idle = !__any_sync(0xffffffffu, mem_ok);   // warps without a cell
    // bits per cell of the quad: updated; of a y face
    unsigned okb = 0, fyb = 0;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        const int y = yq + j;
        if (row_ok && y >= kRadius && y < ny - kRadius) okb |= 1u << j;
        if (y < pml || y >= ny - pml) fyb |= 1u << j;
    }
    Taps T = taps_start(P, rt, q);
    // the x face part, constant along z
    const int fx = x < pml ? 0 : (x >= nx - pml ? 1 : -1);
    const int lix = x < pml ? pml - x : x - nx + pml;
    const bool xy_face = row_ok && (fx >= 0 || (fyb & okb));
    const bool xy_face_warp = __any_sync(0xffffffffu, xy_face);
    // whether the tile reaches into the never-updated band or the row padding
    const bool y_edge = y0 < kRadius || y0 + kTileY > ny - kRadius;
    const float dt = p.dt;
    const float dt2 = __fmul_rn(dt, dt);
    // the reference adds source * wavelet to every cell (CPU_function.c:326-338):
    // a cell without a source gets +-0, which turns a -0 into +0 when the
    // product is +0
    const float zw = __fmul_rn(0.0f, p.wavelet);

    // The cell's own values (u(k-1), the parameters, the PML state) are copied
    // one plane ahead into the thread's slots by cp.async, and read after the
    // stencil: they hold no registers while the stencil runs.
    float4 *own = reinterpret_cast<float4 *>(smem + L.own_off) + tid;
    const int nthr = plane_threads(tile_x);   // a batched CTA may have more
    auto prefetch_params = [&](unsigned b) {
        if (!mem_ok) return;
        if (HALF) {
            cp_async8(own + nthr, p.h_vp + b);
            cp_async8(own + 2 * nthr, p.h_eps + b);
            cp_async8(own + 3 * nthr, p.h_del + b);
        } else {
            cp_async16(own + nthr, p.prm_v + b);
            cp_async16(own + 2 * nthr, p.prm_e + b);
            cp_async16(own + 3 * nthr, p.prm_r + b);
        }
    };
    auto prefetch_u = [&](unsigned b) {
        if (mem_ok) cp_async16(own, p.u_prev + b);
    };
    auto prefetch_pml = [&](unsigned b, bool z_face) {
        if (mem_ok && (xy_face || z_face)) {
            cp_async16(own + 4 * nthr, p.w1o + b);
            cp_async16(own + 5 * nthr, p.w1c + b);
            cp_async16(own + 6 * nthr, p.w3o + b);
            cp_async16(own + 7 * nthr, p.w3c + b);
            cp_async16(own + 8 * nthr, p.po + b);
            cp_async16(own + 9 * nthr, p.pc + b);
            cp_async16(own + 10 * nthr, p.w21o + b);
        }
    };
    auto face_of_z = [&](int z) { return z < pml ? 4 : (z >= nz - pml ? 5 : -1); };
    float mx = 0.0f;
    unsigned base = (unsigned)((long long)z0 * p.plane + (long long)x * p.ldy + yq);
    const unsigned plane = (unsigned)p.plane;

    // Before the previous kernel has finished (grid launches): barriers, the
    // parameters, the layer coefficients and the sources, which no step changes.
    prefetch_params(base);
    if (tid == 0) {
        misc_u[0] = misc_u[1] = 0;   // sources of this column, deferred cells
        pipe_init(P);
    }
    for (int i = tid; i < 3 * pml; i += blockDim.x)
        tab[i] = AR == kArithRef ? p.layers[i] : step_layer(p.layers[i]);
    if (AR == kArithFast && tid < kTileY) {   // layer coefficients of the tile's y cells
        const int y = y0 + tid;
        float4 c = make_float4(0.f, 0.f, 0.f, 0.f);
        if (y < pml) {
            if (y > 0) c = step_layer(p.layers[pml + pml - y]);   // y = 0: never updated
        } else if (y >= ny - pml && y < ny) {
            c = step_layer(p.layers[pml + y - ny + pml]);
            c.w = -c.w;
        }
        ytab[tid] = c.x;
        ytab[kTileY + tid] = c.y;
        ytab[2 * kTileY + tid] = c.z;
        ytab[3 * kTileY + tid] = c.w;
    }
    if (p.nsrc) {   // the sources of this column
        __syncthreads();
        for (int e = tid; e < p.nsrc; e += blockDim.x) {
            const SrcEntry s = p.src[e];
            if (s.x >= x0 && s.x < x0 + tile_x && s.y >= y0 && s.y < y0 + kTileY && s.z >= z0 &&
                s.z < z1)
                csrc[atomicAdd(&misc_u[0], 1u)] = s;
        }
    }
    if (!REUSE) pdl_wait();
    if (tid == 0) pipe_start(P, tm);
    prefetch_u(base);
    if (xy_face_warp || face_of_z(z0) >= 0) prefetch_pml(base, face_of_z(z0) >= 0);
    // The thresholds.  A speculative step finds them where the resolution of
    // the step before left them; otherwise two threads of the last warp work
    // them out while the first loads are on their way.
    if (tid >> 5 == P.ncw - 1 && lane < 2) {
        if (!SPEC) {
            misc[lane] = threshold_m2(p.gmax[p.step]);
        } else if (p.win_ready) {
            misc[lane] = p.win[3 + lane];
        } else {
            float w[3];
            spec_window(p, p.step, p.spec_err, w);
            misc[lane] = threshold_m2(w[lane]);
            if (win_writer && lane == 0) {
                p.win[0] = w[0];
                p.win[1] = w[1];
                p.win[2] = w[2];
            }
        }
    }
    __syncthreads();
    const float T2lo = misc[0], T2hi = misc[1];
    const int ncsrc = (int)misc_u[0];
    bool ok = true;
    // One plane of a warp.  PML: whether a cell of the warp is of the shell.
    // The body exists twice, so that the warps of the interior carry nothing
    // of the shell's update: sharing one body, with the update under a branch,
    // cost them 160 of 650 instructions a plane.
    // reference arithmetic: the classes (window_class) of the thread's quad in
    // the planes staged last, two bits each, the newest lowest
    unsigned zhist = 0;
    float Ux[4], Uy[4], Uz[4], Uxx[4], Uyy[4], Uzz[4], u0[4];
    auto plane_step = [&](int t, auto shell) {
        constexpr bool PML = decltype(shell)::value;
        const int z = z0 + t;
        const int fz = PML ? face_of_z(z) : -1;
        // a thread without a cell reads whatever its slots hold: it stores nothing
        cp_async_wait();
        const float4 u1v = own[0];
        float4 Vv, Ev, Rv;
        if (HALF) {
            quad_params_half(*reinterpret_cast<const uint2 *>(own + nthr),
                             *reinterpret_cast<const uint2 *>(own + 2 * nthr),
                             *reinterpret_cast<const uint2 *>(own + 3 * nthr), Vv, Ev, Rv);
        } else {
            Vv = own[nthr];
            Ev = own[2 * nthr];
            Rv = own[3 * nthr];
        }
        if (t + 1 < nzc) {
            prefetch_u(base + plane);
            prefetch_params(base + plane);
        }
        // |grad u|^2, and the step's own max |grad u|
        float h2[4], m2[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            if (AR == kArithRef) {
                m2[j] = xr::grad_m2(Ux[j], Uy[j], Uz[j]);
                h2[j] = 0.0f;
            } else {
                h2[j] = fmaf(Uy[j], Uy[j], __fmul_rn(Ux[j], Ux[j]));
                m2[j] = fmaf(Uz[j], Uz[j], h2[j]);
            }
        }
        if (SPEC) {   // three-input max: one instruction fewer per cell
            auto add_max = [&](int j) {
                float t2;
                asm("max.f32 %0, %1, %2, %3;" : "=f"(t2) : "f"(mx), "f"(fabsf(Ux[j])), "f"(fabsf(Uy[j])));
                mx = fmaxf(t2, fabsf(Uz[j]));
            };
            if (!y_edge) {   // rows past the tile are left out at the end
                add_max(0); add_max(1); add_max(2); add_max(3);
            } else {
#pragma unroll
                for (int j = 0; j < 4; ++j)
                    if ((okb >> j) & 1u) add_max(j);
            }
        }
        // Scalar operator, GPU_kernel.cu:93-111 / CPU_function.c:339-370.
        // kS: S in the reference arithmetic, (vp dt)^2 S in the fast one; k1:
        // the same with S = 1.  Most warps lie wholly below the threshold
        // (S = 1) or wholly above it; the others decide cell by cell, and
        // list the cells whose decision waits for the exact max.
        float kS[4], k1[4], e1[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            k1[j] = AR == kArithRef ? 1.0f : k_of_vp(f4(Vv, j), dt);
            e1[j] = __fadd_rn(1.0f, f4(Ev, j));
            kS[j] = k1[j];
        }
        unsigned pmlb = 0;   // bits of the quad's PML cells
        if (PML) pmlb = (fx >= 0 || fz >= 0 ? 15u : fyb) & okb;
        unsigned above = 0;
        const bool bits = DEC && (p.dec_in || p.dec_out);   // decisions replayed or kept
        if (bits || !__all_sync(0xffffffffu, !row_ok || max4(m2) <= T2lo)) {
            if (AR == kArithRef) {
#pragma unroll
                for (int j = 0; j < 4; ++j)
                    if (m2[j] > T2lo) above |= 1u << j;
                if (DEC && !SPEC && p.dec_in && row_ok) above = (p.dec_in[base >> 5] >> (4 * q)) & 15u;
#pragma unroll
                for (int j = 0; j < 4; ++j)
                    if ((above & okb) >> j & 1u)
                        kS[j] = scalar_s_call(Ux[j], Uy[j], Uz[j], m2[j], f4(Ev, j), f4(Rv, j));
            } else {
                float S[4];
#pragma unroll
                for (int h = 0; h < 2; ++h) {   // cells (0,1) and (2,3) as pairs
                    const int j0 = 2 * h, j1 = 2 * h + 1;
                    const float2 v = aniso_s2(f2(h2[j0], h2[j1]), f2(m2[j0], m2[j1]),
                                              __fmul2_rn(f2(Uz[j0], Uz[j1]), f2(Uz[j0], Uz[j1])),
                                              f2(f4(Ev, j0), f4(Ev, j1)),
                                              f2(f4(Rv, j0), f4(Rv, j1)));
                    S[j0] = v.x;
                    S[j1] = v.y;
                }
                if (!bits && __all_sync(0xffffffffu, !row_ok || min4(m2) > T2hi)) {
#pragma unroll
                    for (int j = 0; j < 4; ++j) kS[j] = __fmul_rn(k1[j], S[j]);
                } else {
#pragma unroll
                    for (int j = 0; j < 4; ++j)
                        if (m2[j] > T2lo) above |= 1u << j;
                    if (DEC && !SPEC && p.dec_in && row_ok) above = (p.dec_in[base >> 5] >> (4 * q)) & 15u;
#pragma unroll
                    for (int j = 0; j < 4; ++j)
                        kS[j] = (above >> j) & 1u ? __fmul_rn(k1[j], S[j]) : k1[j];
                }
            }
            if (SPEC) {
                unsigned nib = 0;
#pragma unroll
                for (int j = 0; j < 4; ++j)
                    if (!(m2[j] > T2hi)) nib |= 1u << j;
                nib &= above & okb;
                if (__any_sync(0xffffffffu, nib)) {
                    unsigned pos = defer_places(&misc_u[1], nib);
#pragma unroll
                    for (int j = 0; j < 4; ++j) {
                        if (!((nib >> j) & 1u)) continue;
                        if (pos < seg.cap) {
                            const size_t e = seg.base + pos;
                            p.dkey[e] = make_uint2(base + j, __float_as_uint(m2[j]));
                            float4 v;
                            if ((pmlb >> j) & 1u) {
                                const int f = fx >= 0 ? fx : ((fyb >> j) & 1u ? 2 : 4);
                                v = pml_inputs<AR>(f, e1[j], Ux[j], Uy[j], Uz[j], Uxx[j], Uyy[j],
                                                   Uzz[j]);
                            } else {
                                v.x = interior_cell<AR>(u0[j], f4(u1v, j), Uxx[j], Uyy[j], Uzz[j],
                                                        e1[j], k1[j], f4(Vv, j), dt2);
                            }
                            p.dval[e] = v;
                        }
                        ++pos;
                    }
                }
            }
        }
        float out[4];
#pragma unroll
        for (int j = 0; j < 4; ++j)
            out[j] = interior_cell<AR>(u0[j], f4(u1v, j), Uxx[j], Uyy[j], Uzz[j], e1[j], kS[j],
                                       f4(Vv, j), dt2);
        if (PML) {
            if (xy_face || (row_ok && fz >= 0)) {
                PmlOwn o;
                o.w11 = own[4 * nthr]; o.w12 = own[5 * nthr];
                o.w31 = own[6 * nthr]; o.w32 = own[7 * nthr];
                o.p1 = own[8 * nthr];  o.p2 = own[9 * nthr];
                o.w21 = own[10 * nthr];
                if (t + 1 < nzc) prefetch_pml(base + plane, face_of_z(z + 1) >= 0);
                PmlNew n;
                const int liz = z < pml ? pml - z : z - nz + pml;
                if (AR == kArithRef)
                    pml_quad_ref(p, tab, kS, e1, Vv, Ux, Uy, Uz, Uxx, Uyy, Uzz, o, pmlb, fx, lix,
                                 yq, fz, liz, out, n);
                else
                    pml_quad_fast(p, tab, ytab + 4 * q, kS, e1, Ux, Uy, Uz, Uxx, Uyy, Uzz, o, pmlb,
                                  fyb, fx, lix, fz, liz, out, n);
                if (mem_ok) {
                    *reinterpret_cast<float4 *>(p.w1n + base) = make_float4(n.w13[0].x, n.w13[0].y, n.w13[1].x, n.w13[1].y);
                    *reinterpret_cast<float4 *>(p.w3n + base) = make_float4(n.w33[0].x, n.w33[0].y, n.w33[1].x, n.w33[1].y);
                    *reinterpret_cast<float4 *>(p.pn + base) = make_float4(n.p3[0].x, n.p3[0].y, n.p3[1].x, n.p3[1].y);
                    *reinterpret_cast<float4 *>(p.w21n + base) = make_float4(n.w21[0].x, n.w21[0].y, n.w21[1].x, n.w21[1].y);
                }
            }
        }
        // a quad of the shell has asked for the next plane's state already
        // (as soon as it had read its own: 2.5 % of a step on 240x240x190
        // against here)
        if (t + 1 < nzc && face_of_z(z + 1) >= 0 && !(PML && (xy_face || (row_ok && fz >= 0))))
            prefetch_pml(base + plane, true);
        if (AR == kArithRef) {   // source injection (CPU_function.c:334): u3 += source * wavelet
            unsigned srcb = 0;
            for (int e = 0; e < ncsrc; ++e) {
                const SrcEntry s = csrc[e];
                if (s.z == z && s.x == x) {
                    const float add = __fmul_rn(s.v, p.wavelet);
#pragma unroll
                    for (int j = 0; j < 4; ++j)
                        if (s.y - yq == j) {
                            out[j] = __fadd_rn(out[j], add);
                            srcb |= 1u << j;
                        }
                }
            }
#pragma unroll
            for (int j = 0; j < 4; ++j)
                if (!((srcb >> j) & 1u)) out[j] = __fadd_rn(out[j], zw);
        }
        if (y_edge) {
#pragma unroll
            for (int j = 0; j < 4; ++j) out[j] = (okb >> j) & 1u ? out[j] : u0[j];   // never updated
        }
        if (mem_ok)
            *reinterpret_cast<float4 *>(p.u_out + base) = make_float4(out[0], out[1], out[2], out[3]);
        // the step's decisions, when asked for: one bit per cell, 32 y cells a
        // word (the 8 lanes of a row combine their 4 bits)
        if (DEC && p.dec_out) {
            unsigned w = (above & okb) << (4 * q);
            w |= __shfl_xor_sync(0xffffffffu, w, 1);
            w |= __shfl_xor_sync(0xffffffffu, w, 2);
            w |= __shfl_xor_sync(0xffffffffu, w, 4);
            if (q == 0 && row_ok) p.dec_out[base >> 5] = w;
        }
        pipe_release(P, tm, t);
    };
    for (int t = 0; t < nzc; taps_next(T, P, t), ++t, base += plane) {
        ok = __all_sync(0xffffffffu, pipe_wait(P, t));   // warps stay converged for the collectives below
        if (!ok) break;
        if (idle) {
            pipe_release(P, tm, t);
            continue;
        }
        if (AR == kArithRef) {
            if (t == 0)
                for (int i = 0; i < 2 * kRadius; ++i) zhist = (zhist << 2) | window_class(ztap(T, i));
            zhist = (zhist << 2) | window_class(ztap(T, 2 * kRadius));
            unsigned cls = halo_class(T.pc - ((rt + kRadius) * kBoxY + kHaloY + 4 * q), r & ~3, tile_x);
            if (row_ok) cls |= ((zhist & 0x155555u) ? 1u : 0u) | ((zhist & 0x2aaaaau) ? 2u : 0u);
            cls = k.div_ok ? __reduce_or_sync(0xffffffffu, cls) : 2u;
            if (cls == 0) quad_derivs_ref(T, k, Ux, Uy, Uz, Uxx, Uyy, Uzz, u0);
            else if (cls == 1) quad_derivs_ref_loop<kDivScaled>(T, k, Ux, Uy, Uz, Uxx, Uyy, Uzz, u0);
            else quad_derivs_ref_loop<kDivIeee>(T, k, Ux, Uy, Uz, Uxx, Uyy, Uzz, u0);
        } else {
            quad_derivs<true>(T, k, Ux, Uy, Uz, Uxx, Uyy, Uzz, u0);
        }
        if (xy_face_warp || face_of_z(z0 + t) >= 0) plane_step(t, std::true_type());
        else plane_step(t, std::false_type());
    }
    cp_async_wait();
    // What happens on one plane only stays out of the loop; each thread works
    // on the cells it has just written.  Source injection (GPU_kernel.cu:727):
    // u3 += source * wavelet.
    if (AR == kArithFast && ok)
        for (int e = 0; e < ncsrc; ++e) {
            const SrcEntry s = csrc[e];
            if (s.x == x && (unsigned)(s.y - yq) < 4u) {
                float *u = p.u_out + ((long long)s.z * p.plane + (long long)x * p.ldy + s.y);
                *u = __fadd_rn(*u, __fmul_rn(s.v, p.wavelet));
            }
        }
    // receiver plane (3dPureqPModeling_single_shot.cu:333-337)
    if (p.record && ok && p.sz >= z0 && p.sz < z1 && mem_ok && x >= pml && x < nx - pml) {
        const float4 u = *reinterpret_cast<const float4 *>(
            p.u_out + ((long long)p.sz * p.plane + (long long)x * p.ldy + yq));
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const int y = yq + j;
            if (((okb >> j) & 1u) && y >= pml && y < ny - pml)
                p.record[(long long)(x - pml) * (ny - 2 * pml) + (y - pml)] = f4(u, j);
        }
    }
    ok = pipe_finish(P, ok, p.err);
    if (SPEC) {
        if (!row_ok) mx = 0.0f;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
        if (lane == 0 && mx > 0.0f &&
            mx > *reinterpret_cast<const volatile float *>(p.gmax + p.step))
            atomicMax(reinterpret_cast<unsigned *>(p.gmax + p.step), __float_as_uint(mx));
        if (tid == 0) {
            *seg.count = misc_u[1];
            if (misc_u[1] > seg.cap) *const_cast<int *>(p.gate) = 1;   // re-run the step
        }
    }
    if (REUSE && tid == 0 && ok) pipe_inval(P);
    return ok;
}

template <bool SPEC, bool HALF, int AR, bool DEC = !SPEC>
__global__ void __launch_bounds__(kStepThreads, 2)
    qp3d_step_kernel(const __grid_constant__ TileMaps tm, const PlaneParams p)
{
    extern __shared__ __align__(128) unsigned char smem[];
    pdl_trigger();
    const int y0 = blockIdx.x * kTileY, x0 = kRadius + blockIdx.y * p.tile_x;
    const int z0 = kRadius + blockIdx.z * p.chunk_z;
    const int z1 = min(z0 + p.chunk_z, p.nz - kRadius);
    if (z0 >= z1) {
        pdl_wait();
        return;
    }
    const unsigned id = blockIdx.x + gridDim.x * (blockIdx.y + gridDim.y * blockIdx.z);
    const DeferSeg seg = {(size_t)id * p.dcap, p.dcap, p.dcount + id};
    step_tile<SPEC, false, HALF, AR, DEC>(&tm, p, p.k, p.tile_x, y0, x0, z0, z1, id == 0, seg,
                                          smem);
}

// ---------------------------------------------------------------------------
// Resolution of a speculative step, once its step kernel has finished and the
// true max M of the step is known.  M outside the predicted window, or a
// segment that ran over: the step is re-run exactly.  Otherwise every listed
// cell that turns out to be below the threshold of M gets the S = 1 results
// the step kernel stored for it.
// ---------------------------------------------------------------------------
__device__ __forceinline__ bool step_missed(const PlaneParams &p)
{
    const float M = p.gmax[p.step];
    return !((M >= p.win[0]) && (M <= p.win[1])) || *p.gate != 0;
}

// The re-run flag of the step and the history of the prediction's relative
// errors (one warp of the grid; lanes 0 and 1), and, for the shots of a single
// launch (p.win_next), the window and the thresholds of the next step.
// Threads that read the flag meanwhile come to the same step_missed either
// way.
__device__ __forceinline__ void step_account(const PlaneParams &p, float *spec_err)
{
    const int lane = threadIdx.x & 31;
    const float M = p.gmax[p.step], pred = p.win[2];
    const bool missed = step_missed(p);
    float err[kSpecHist];
#pragma unroll
    for (int i = kSpecHist - 1; i > 0; --i) err[i] = spec_err[i - 1];
    err[0] = pred > 0.0f ? fabsf(__fdiv_rn(M, pred) - 1.0f) : 1.0f;
    __syncwarp(3u);
    if (lane == 0) {
        if (missed) *const_cast<int *>(p.gate) = 1;
#pragma unroll
        for (int i = 0; i < kSpecHist; ++i) spec_err[i] = err[i];
    }
    if (!p.win_next) return;
    float w[3];
    spec_window(p, p.step + 1, err, w);
    p.win_next[3 + lane] = threshold_m2(w[lane]);
    p.win_next[lane] = w[lane];
    if (lane == 0) p.win_next[2] = w[2];
}

// S = 1 results of entry e, if its cell is below the threshold
// (double)mode > 0.01 * (double)max  <=>  mode > Tf (see threshold_m2).
template <bool HALF, int AR>
__device__ __forceinline__ void fix_cell(const PlaneParams &p, float Tf, size_t e)
{
    const uint2 key = p.dkey[e];
    const float4 v = p.dval[e];
    if (__fsqrt_rn(__uint_as_float(key.y)) > Tf) return;
    const int nx = p.nx, ny = p.ny, nz = p.nz, pml = p.pml;
    const unsigned plane = (unsigned)p.plane, ldy = (unsigned)p.ldy, idx = key.x;
    const int z = (int)(idx / plane);
    const unsigned rem = idx - (unsigned)z * plane;
    const int x = (int)(rem / ldy), y = (int)(rem - (unsigned)x * ldy);
    const int fx = x < pml ? 0 : (x >= nx - pml ? 1 : -1);
    const int fy = y < pml ? 2 : (y >= ny - pml ? 3 : -1);
    const int fz = z < pml ? 4 : (z >= nz - pml ? 5 : -1);
    float out = v.x;
    if (fx >= 0 || fy >= 0 || fz >= 0) {
        int f, li;
        cell_face(fx, x < pml ? pml - x : x - nx + pml, fy, y < pml ? pml - y : y - ny + pml, fz,
                  z < pml ? pml - z : z - nz + pml, f, li);
        float vp, e1;
        if (HALF) {
            vp = __half2float(p.h_vp[idx]);
            e1 = __fadd_rn(1.0f, __fmul_rn(2.0f, __half2float(p.h_eps[idx])));
        } else {
            vp = p.prm_v[idx];
            e1 = __fadd_rn(1.0f, p.prm_e[idx]);
        }
        const xr::PmlOut o = pml_cell<AR>(
            f, p.layers[(f >> 1) * pml + li], AR == kArithRef ? 1.0f : k_of_vp(vp, p.dt), e1, vp,
            v, p.dt, p.w1o[idx], p.w1c[idx], p.w21o[idx], p.w3o[idx], p.w3c[idx], p.po[idx],
            p.pc[idx]);
        p.w1n[idx] = o.w13;
        p.w21n[idx] = o.w21;
        p.w3n[idx] = o.w33;
        p.pn[idx] = o.p3;
        out = o.u3;
    }
    bool has_src = false;
    for (int i = 0; i < p.nsrc; ++i) {
        const SrcEntry s = p.src[i];
        if (s.z == z && s.x == x && s.y == y) {
            out = __fadd_rn(out, __fmul_rn(s.v, p.wavelet));
            has_src = true;
        }
    }
    if (AR == kArithRef && !has_src) out = __fadd_rn(out, __fmul_rn(0.0f, p.wavelet));
    p.u_out[idx] = out;
    if (p.dec_out) atomicAnd(p.dec_out + (idx >> 5), ~(1u << (idx & 31)));
    if (p.record && z == p.sz && x >= pml && x < nx - pml && y >= pml && y < ny - pml)
        p.record[(long long)(x - pml) * (ny - 2 * pml) + (y - pml)] = out;
}

// A block's share of the segments, kThreads at a time: their lengths (count)
// are scanned to offsets, so that the threads share the cells evenly however
// the lengths differ.  len(i, n) is how many of segment i's n cells to fix (0:
// none), fix(i, j) handles its entry j.
template <class Len, class Fix>
__device__ __forceinline__ void for_segment_cells(int nseg, const unsigned *count, Len len, Fix fix)
{
    __shared__ unsigned s_off[kThreads + 1], s_w[kThreads / 32];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, nw = blockDim.x >> 5;
    for (int first = 0; first * (int)gridDim.x + (int)blockIdx.x < nseg; first += blockDim.x) {
        const long long i = blockIdx.x + (long long)(first + tid) * gridDim.x;
        const unsigned n = i < nseg ? count[i] : 0u;   // beside the loads len asks for
        const unsigned c = i < nseg ? len((int)i, n) : 0u;
        unsigned incl = c;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const unsigned v = __shfl_up_sync(0xffffffffu, incl, o);
            if (lane >= o) incl += v;
        }
        if (lane == 31) s_w[warp] = incl;
        __syncthreads();
        unsigned add = 0, total = 0;
        for (int w = 0; w < nw; ++w) {
            if (w < warp) add += s_w[w];
            total += s_w[w];
        }
        s_off[tid + 1] = add + incl;
        if (tid == 0) s_off[0] = 0;
        __syncthreads();
        for (unsigned e = tid; e < total; e += blockDim.x) {
            int lo = 0, hi = blockDim.x;   // s_off[lo] <= e < s_off[hi]
            while (hi - lo > 1) {
                const int m = (lo + hi) >> 1;
                if (s_off[m] <= e) lo = m;
                else hi = m;
            }
            fix((int)(blockIdx.x + (long long)(first + lo) * gridDim.x), e - s_off[lo]);
        }
        __syncthreads();
    }
}

__device__ __forceinline__ float threshold_of(float gmax)
{
    return __double2float_rd(1.0e-02 * (double)gmax);
}

// Resolution of a single shot's speculative step: a persistent grid of two
// CTAs per SM, held to the registers that leave room for a CTA of the next
// step beside them.  The re-run takes the step's tile columns in turn, so a step
// that needs none costs one short wave instead of a full grid of CTAs that
// each read the flag and exit.
template <bool HALF, int AR>
__global__ void __launch_bounds__(kStepThreads, 2)
    qp3d_fix_or_rerun_kernel(const __grid_constant__ TileMaps tm, const PlaneParams p,
                             float *spec_err)
{
    pdl_trigger();
    pdl_wait();
    const int nyt = (p.ny - kRadius - 1) / kTileY + 1;
    const int nxt = (p.nx - 2 * kRadius + p.tile_x - 1) / p.tile_x;
    const int nch = (p.nz - 2 * kRadius + p.chunk_z - 1) / p.chunk_z;
    const int ntiles = nyt * nxt * nch;
    if (blockIdx.x == gridDim.x - 1 && threadIdx.x < 2) step_account(p, spec_err);
    for_segment_cells(
        ntiles, p.dcount,
        [&](int, unsigned n) {
            if (n) atomicAdd(p.alt_count, n);
            return step_missed(p) ? 0u : n;
        },
        [&](int i, unsigned j) {
            fix_cell<HALF, AR>(p, threshold_of(p.gmax[p.step]), (size_t)i * p.dcap + j);
        });
    if (!step_missed(p)) return;
    extern __shared__ __align__(128) unsigned char smem[];
    const DeferSeg none = {0, 0, nullptr};
    for (int t = blockIdx.x; t < ntiles; t += gridDim.x) {
        const int by = t % nyt, bx = (t / nyt) % nxt, bz = t / (nyt * nxt);
        const int z0 = kRadius + bz * p.chunk_z;
        const int z1 = min(z0 + p.chunk_z, p.nz - kRadius);
        if (z0 >= z1) continue;
        if (!step_tile<false, true, HALF, AR, true>(&tm, p, p.k, p.tile_x, by * kTileY,
                                                    kRadius + bx * p.tile_x, z0, z1, false, none,
                                                    smem))
            return;
    }
}

// ---------------------------------------------------------------------------
// Small kernels
// ---------------------------------------------------------------------------

// Sources outside the updated box [5,n-5)^3: the reference never updates
// those cells, so u3 there is its previous value plus the source
// (CPU_function.c:326-338 on a cell wavefield_update skips); with two
// buffers that previous value is u(k).
__global__ void qp3d_band_source_kernel(float *u_new, const float *u_cur, const SrcEntry *src,
                                        int n, long long plane, int ldy, float w)
{
    int e = blockIdx.x * blockDim.x + threadIdx.x;
    if (e >= n) return;
    SrcEntry s = src[e];
    long long i = (long long)s.z * plane + (long long)s.x * ldy + s.y;
    u_new[i] = __fadd_rn(u_cur[i], __fmul_rn(s.v, w));
}

// All sources, after the step kernel (used when there are too many to fuse).
__global__ void qp3d_all_source_kernel(float *u_new, const float *u_cur, const SrcEntry *src,
                                       int n, long long plane, int ldy, int nx, int ny, int nz,
                                       float w)
{
    int e = blockIdx.x * blockDim.x + threadIdx.x;
    if (e >= n) return;
    SrcEntry s = src[e];
    long long i = (long long)s.z * plane + (long long)s.x * ldy + s.y;
    bool inside = s.x >= kRadius && s.x < nx - kRadius && s.y >= kRadius && s.y < ny - kRadius &&
                  s.z >= kRadius && s.z < nz - kRadius;
    float prev = inside ? u_new[i] : u_cur[i];
    u_new[i] = __fadd_rn(prev, __fmul_rn(s.v, w));
}

__global__ void qp3d_record_kernel(const float *u, float *rec, int nx, int ny, int pml, int sz,
                                   int ldy, long long plane)
{
    int hx = nx - 2 * pml, hy = ny - 2 * pml;
    long long n = (long long)hx * hy;
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n;
         i += (long long)gridDim.x * blockDim.x) {
        int xi = (int)(i / hy), yi = (int)(i % hy);
        rec[i] = u[(long long)sz * plane + (long long)(xi + pml) * ldy + yi + pml];
    }
}

__global__ void qp3d_crop_kernel(const float *u, float *out, int x0, int x1, int y0, int y1,
                                 int z0, int z1, int ldy, long long plane)
{
    long long nyc = y1 - y0, nxc = x1 - x0, nzc = z1 - z0;
    long long n = nxc * nyc * nzc;
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n;
         i += (long long)gridDim.x * blockDim.x) {
        long long yi = i % nyc, xi = (i / nyc) % nxc, zi = i / (nyc * nxc);
        out[i] = u[(zi + z0) * plane + (xi + x0) * ldy + yi + y0];
    }
}

// Per-cell parameters vp, 2 eps, 8 (eps - delta) from dense [nz][nx][ny]
// volumes (the caller's layout) into the pitched layout, one thread per
// pitched cell, row padding zero; and the same layout change for
// half-precision storage.
__global__ void qp3d_params_dense_kernel(const float *vp, const float *eps, const float *del,
                                         float *VP, float *E2, float *R8, int ny,
                                         long long vol, int ldy)
{
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < vol;
         i += (long long)gridDim.x * blockDim.x) {
        const long long row = i / ldy;
        const int y = (int)(i - row * ldy);
        float v = 0.0f, e2 = 0.0f, r8 = 0.0f;
        if (y < ny) {
            const long long j = row * ny + y;
            const float e = eps[j], d = del[j];
            v = vp[j];
            e2 = __fmul_rn(2.0f, e);
            r8 = __fmul_rn(8.0f, __fsub_rn(e, d));
        }
        VP[i] = v;
        E2[i] = e2;
        R8[i] = r8;
    }
}

__global__ void qp3d_to_half_dense_kernel(const float *a, __half *h, int ny, long long vol,
                                          int ldy)
{
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < vol;
         i += (long long)gridDim.x * blockDim.x) {
        const long long row = i / ldy;
        const int y = (int)(i - row * ldy);
        h[i] = __float2half_rn(y < ny ? a[row * ny + y] : 0.0f);
    }
}

// ---------------------------------------------------------------------------
// Batched shots.  Per time step:
//   qp3d_batch_prepare_kernel   reads the step counter k, writes every shot's
//                               PlaneParams of step k (buffer rotation,
//                               wavelet[k], record plane, per-step slots),
//                               zeroes the re-run queue, sets the counter to
//                               k + 1.  The step is therefore the same
//                               sequence of launches for every k and can be
//                               captured once in a CUDA graph.
//   qp3d_batch_plane_kernel     one CTA per work item -- one tile column of
//                               one shot -- runs the gradmax or step tile
//                               body on it; uneven shot sizes mix in one
//                               launch.
//   qp3d_batch_resolve_kernel   the resolution of a speculative step.
// ---------------------------------------------------------------------------
__global__ void qp3d_batch_prepare_kernel(const BatchShot *shots, int nshots, PlaneParams *pp,
                                          int *ctr, int *queue, int spec)
{
    pdl_trigger();
    pdl_wait();
    const int k = *ctr;
    for (int s = threadIdx.x; s < nshots; s += blockDim.x) {
        const BatchShot &b = shots[s];
        PlaneParams p;
        memset(&p, 0, sizeof(p));
        p.nx = b.nx; p.ny = b.ny; p.nz = b.nz; p.ldy = b.ldy; p.pml = b.pml; p.sz = b.sz;
        p.plane = b.plane;
        p.dt = b.dt;
        p.step = k;
        p.err = b.err;
        p.active = k < b.nt ? 1 : 0;
        if (p.active) {
            // the host's rotation of qp3d_shot_advance from a reset shot
            const int a = (3 - k % 3) % 3, bb = (a + 1) % 3, c = (a + 2) % 3;
            p.ucur = a;
            p.u_cur = b.U[a]; p.u_prev = b.U[bb]; p.u_out = b.U[c];
            p.prm_v = b.VP; p.prm_e = b.E2; p.prm_r = b.R8;
            const int lo = k % 3, lc = (k + 1) % 3, ln = (k + 2) % 3;
            p.w1o = b.W1[lo]; p.w1c = b.W1[lc]; p.w1n = b.W1[ln];
            p.w3o = b.W3[lo]; p.w3c = b.W3[lc]; p.w3n = b.W3[ln];
            p.po = b.P[lo];   p.pc = b.P[lc];   p.pn = b.P[ln];
            p.w21o = b.W21[k % 2];
            p.w21n = b.W21[(k + 1) % 2];
            p.layers = b.layers;
            p.gmax = b.gmax;
            p.record = b.record + (long long)k * b.hx * b.hy;
            p.src = b.src;
            p.nsrc = b.nsrc;
            p.wavelet = b.wavelet[k];
            p.spec = spec;
            p.gate = spec ? b.redo + k : nullptr;
            p.win = b.win + kWinFloats * (long long)k;
            p.spec_err = b.spec_err;
            p.delta_min = b.delta_min;
            p.spec_bias = b.spec_bias;
            p.dkey = b.dkey;
            p.dval = b.dval;
            p.alt_count = b.alt_count + k;
            if (spec) {
                float w[3];
                spec_window(p, k, p.spec_err, w);
                p.win[0] = w[0];
                p.win[1] = w[1];
                p.win[2] = w[2];
                p.win[3] = threshold_m2(w[0]);
                p.win[4] = threshold_m2(w[1]);
                p.win_ready = 1;
            }
        }
        pp[s] = p;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        *queue = 0;
        *ctr = k + 1;
    }
}

constexpr size_t kParamBytes = (sizeof(PlaneParams) + 127) & ~(size_t)127;

size_t batch_smem_bytes(int tile_x, int pml, int nsrc)
{
    return kParamBytes + plane_smem_bytes(tile_x, pml, nsrc);
}

// One work item: KIND 0 gradmax, 1 exact step, 2 speculative step.  sp: a copy
// of the shot's parameters in shared memory.
template <int KIND, bool REUSE, int AR>
__device__ __forceinline__ bool batch_item(const BatchArgs &b, int it, unsigned char *smem)
{
    PlaneParams *sp = reinterpret_cast<PlaneParams *>(smem);
    unsigned char *body = smem + kParamBytes;
    const WorkItem w = b.work[it];
    {
        const unsigned *src = reinterpret_cast<const unsigned *>(b.pp + w.shot);
        unsigned *dst = reinterpret_cast<unsigned *>(sp);
        for (int i = threadIdx.x; i < (int)(sizeof(PlaneParams) / 4); i += blockDim.x)
            dst[i] = src[i];
    }
    const TileMaps *tm = b.tm + 3 * w.shot;
    if (threadIdx.x == 0)   // maps written by the host before the launch
        for (int i = 0; i < 3; ++i) {
            asm volatile("fence.proxy.tensormap::generic.acquire.gpu [%0], 128;" ::"l"(&tm[i].z)
                         : "memory");
            asm volatile("fence.proxy.tensormap::generic.acquire.gpu [%0], 128;" ::"l"(&tm[i].c)
                         : "memory");
        }
    __syncthreads();
    const PlaneParams &p = *sp;
    tm += p.ucur;
    if (KIND == 0) {
        float mx;
        const bool ok = gradmax_tile<AR>(tm, p, b.k, w.tile_x, w.y0, w.x0, w.z0, w.z1, body, mx);
        gradmax_publish(p, mx);
        return ok;
    }
    const bool first = w.y0 == 0 && w.x0 == kRadius && w.z0 == kRadius;
    const DeferSeg seg = {w.dbase, w.dcap, b.dcount + it};
    return step_tile<KIND == 2, REUSE, false, AR, false>(tm, p, b.k, w.tile_x, w.y0, w.x0, w.z0,
                                                         w.z1, first, seg, body);
}

// All items of a step, one per CTA, longest columns first.
template <int KIND, int AR>
__global__ void __launch_bounds__(kStepThreads, 2)
    qp3d_batch_plane_kernel(const __grid_constant__ BatchArgs b)
{
    extern __shared__ __align__(128) unsigned char smem[];
    pdl_trigger();
    pdl_wait();
    if (b.pp[b.work[blockIdx.x].shot].active) batch_item<KIND, false, AR>(b, blockIdx.x, smem);
}

// After a speculative step of all shots: the resolution of every shot, then
// the exact step of those that missed, by persistent CTAs that take the items
// from a queue (most steps have none).
template <int AR>
__global__ void __launch_bounds__(kStepThreads, 2)
    qp3d_batch_resolve_kernel(const __grid_constant__ BatchArgs b)
{
    extern __shared__ __align__(128) unsigned char smem[];
    // item slot double-buffered by iteration: thread 0 can run one iteration
    // ahead of the others only on the skip path, which has no second barrier
    __shared__ int s_item[2], s_run[2], s_missed;
    pdl_trigger();
    pdl_wait();
    if (threadIdx.x == 0) s_missed = 0;
    __syncthreads();
    if (blockIdx.x == gridDim.x - 1 && threadIdx.x < 2)
        for (int s = 0; s < b.nshots; ++s)
            if (b.pp[s].active) step_account(b.pp[s], const_cast<float *>(b.pp[s].spec_err));
    for (int s = threadIdx.x; s < b.nshots; s += blockDim.x)
        if (b.pp[s].active && step_missed(b.pp[s])) s_missed = 1;
    for_segment_cells(
        b.nwork, b.dcount,
        [&](int i, unsigned n) {
            const PlaneParams &g = b.pp[b.work[i].shot];
            if (!g.active) return 0u;
            if (n) atomicAdd(g.alt_count, n);
            return n && !step_missed(g) ? n : 0u;
        },
        [&](int i, unsigned j) {
            const PlaneParams &g = b.pp[b.work[i].shot];
            fix_cell<false, AR>(g, threshold_of(g.gmax[g.step]), b.work[i].dbase + j);
        });
    __syncthreads();
    if (!s_missed) return;
    for (int iter = 0;; ++iter) {
        const int slot = iter & 1;
        if (threadIdx.x == 0) {
            const int it = atomicAdd(b.queue, 1);
            int run = 0;
            if (it < b.nwork) {
                const PlaneParams &g = b.pp[b.work[it].shot];
                run = g.active && step_missed(g);
            }
            s_item[slot] = it;
            s_run[slot] = run;
        }
        __syncthreads();
        const int it = s_item[slot];
        if (it >= b.nwork) return;
        if (s_run[slot] && !batch_item<1, true, AR>(b, it, smem)) return;
    }
}

// ---------------------------------------------------------------------------
// Adjoint (qp3d_adjoint.cu drives them).  Pass A, per cell: the residual of
// the step is injected at the receivers; the scalar operator of step k is
// rebuilt from u^k (its decision is the forward's; its dependence on eps, delta
// and, with the live operator, the unit normal is differentiated); the PML
// recursions and the interior leapfrog are transposed term by term; each
// derivative the update took of u^k leaves a coefficient field; the gradient
// terms lambda * (d update / d m) are summed.  Pass B, per cell: the transposed
// stencils of the six coefficient fields (second derivatives: the stencil
// itself; first derivatives: its negative), zero outside the volume.
// Pass A writes the quads with updated cells: the adjoint of u, Cxx and Czz; Cyy
// where it can differ from Cxx; Cx, Cy, Cz with the live operator, otherwise
// where a cell is of the shell, as the PML state.  (The adjoint of u_prev is not
// kept, see AdjParams.)  The caller zeroes every buffer once, so the entries
// never written stay zero in all buffers that take turns.
// The gradient is checked against the FP64 adjoint by cosine, not bit for
// bit, so these kernels take the cheaper arithmetic: fast division
// (__fdividef, 2 ulp) in S and its derivatives, fused multiply-adds in the
// transposed stencils.  Pass A is bound by HBM, pass B by the latency of the
// taps it gathers through L1 (see each).
// ---------------------------------------------------------------------------
__device__ __forceinline__ float4 ldg4_or0(const float *f, long long j, bool ok)
{
    return ok ? __ldg(reinterpret_cast<const float4 *>(f + j)) : make_float4(0.f, 0.f, 0.f, 0.f);
}

// The 20 values y-8 .. y+11 of a field around a quad (zero off the row).
__device__ __forceinline__ void row_window(const float *f, long long i, int y, int ldy, float w[20])
{
#pragma unroll
    for (int b = 0; b < 5; ++b) {
        const int yb = y - 8 + 4 * b;
        const float4 v = ldg4_or0(f, i - 8 + 4 * b, yb >= 0 && yb < ldy);
        w[4 * b] = v.x; w[4 * b + 1] = v.y; w[4 * b + 2] = v.z; w[4 * b + 3] = v.w;
    }
}

// Derivatives of u^k for pass A, two cells at a time.  The second derivatives
// keep the centre weight in one coefficient.
__device__ __forceinline__ void adj_derivs(const Taps &T, const Coefs &k, float Ux[4], float Uy[4],
                                           float Uz[4], float Uxx[4], float Uyy[4], float Uzz[4])
{
    const float *pc = T.pc;
    float Y[20];
#pragma unroll
    for (int b = 0; b < 5; ++b) {
        const float4 v = lds4(pc - 8 + 4 * b);
        Y[4 * b] = v.x; Y[4 * b + 1] = v.y; Y[4 * b + 2] = v.z; Y[4 * b + 3] = v.w;
    }
    const float2 uc[2] = {f2(Y[8], Y[9]), f2(Y[10], Y[11])};
#pragma unroll
    for (int h = 0; h < 2; ++h) {
        const int j0 = 2 * h, j1 = j0 + 1;
        float2 g = f2(0.f, 0.f), l = __fmul2_rn(k.ky2, uc[h]);
#pragma unroll
        for (int m = 0; m < kRadius; ++m) {
            const float2 a = f2(Y[8 + j0 + m + 1], Y[8 + j1 + m + 1]);
            const float2 b = f2(Y[8 + j0 - m - 1], Y[8 + j1 - m - 1]);
            const float2 d = sub2(a, b);
            g = m == 0 ? __fmul2_rn(k.cy2[0], d) : __ffma2_rn(k.cy2[m], d, g);
            l = __ffma2_rn(k.c2y2[m], __fadd2_rn(a, b), l);
        }
        Uy[j0] = g.x; Uy[j1] = g.y;
        Uyy[j0] = l.x; Uyy[j1] = l.y;
    }
#pragma unroll
    for (int ax = 0; ax < 2; ++ax) {   // x, then z
        const float2 kc = ax ? k.kz2 : k.kx2;
        float2 g[2] = {f2(0.f, 0.f), f2(0.f, 0.f)};
        float2 l[2] = {__fmul2_rn(kc, uc[0]), __fmul2_rn(kc, uc[1])};
#pragma unroll
        for (int m = 0; m < kRadius; ++m) {
            const float4 a = ax ? ztap(T, kRadius + m + 1) : lds4(pc + (m + 1) * kBoxY);
            const float4 b = ax ? ztap(T, kRadius - m - 1) : lds4(pc - (m + 1) * kBoxY);
            const float2 c1 = ax ? k.cz2[m] : k.cx2[m], c2 = ax ? k.c2z2[m] : k.c2x2[m];
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const float2 d = sub2(half2of(a, h), half2of(b, h));
                g[h] = m == 0 ? __fmul2_rn(c1, d) : __ffma2_rn(c1, d, g[h]);
                l[h] = __ffma2_rn(c2, __fadd2_rn(half2of(a, h), half2of(b, h)), l[h]);
            }
        }
        float *U = ax ? Uz : Ux, *UU = ax ? Uzz : Uxx;
        U[0] = g[0].x; U[1] = g[0].y; U[2] = g[1].x; U[3] = g[1].y;
        UU[0] = l[0].x; UU[1] = l[0].y; UU[2] = l[1].x; UU[3] = l[1].y;
    }
}

// Pass A, marching along z as the step kernels do: u^k staged by TMA, the
// cell's own values copied one plane ahead by cp.async, four consecutive y
// cells (a quad) per thread, a loop body of its own for the warps with cells
// of the shell.  Bound by HBM: 72 bytes a cell of the interior.  (One thread
// per quad that gathered its 31 taps through L1 held 128 registers with
// spills, and waited for three dependent groups of loads: 258 us on
// 240x240x190, 50% of the DRAM peak; this form 199 us with the 80 bytes of
// storing u_prev's adjoint and Cyy as well, 189 now.  Without the stencil it
// takes 200, without the stores of the six fields 150.)  Only updated cells are
// written: the adjoint of the never-updated band reaches no other cell and no
// output.
constexpr int kAdjStreams = 15;
constexpr int kAdjThreads = kQuadsY * kAdjTileX;

#define QP3D_ST4(ptr, v) *reinterpret_cast<float4 *>((ptr) + base) = make_float4(v[0], v[1], v[2], v[3])
__global__ void __launch_bounds__(kAdjThreads, 2)
    qp3d_adj_a_kernel(const __grid_constant__ TileMaps tm, const AdjParams a)
{
    extern __shared__ __align__(128) unsigned char smem[];
    pdl_trigger();
    const int tile_x = a.tile_x;
    const int y0 = blockIdx.x * kTileY, x0 = kRadius + blockIdx.y * tile_x;
    const int z0 = kRadius + blockIdx.z * a.chunk_z, z1 = min(z0 + a.chunk_z, a.nz - kRadius);
    if (z0 >= z1) {
        pdl_wait();
        return;
    }
    const int tid = threadIdx.x;
    const int q = tid & (kQuadsY - 1), r = tid / kQuadsY;
    const int nzc = z1 - z0, nx = a.nx, ny = a.ny, nz = a.nz, pml = a.pml;
    const SmemLayout L = smem_layout(tile_x, pml, 0, kAdjStreams);
    float4 *tab = reinterpret_cast<float4 *>(smem + L.tab_off);
    Pipe<kGroups> P;
    pipe_setup(P, smem, L, tile_x, y0, x0, z0, nzc);
    pipe_hooks(P, a.wait_ns, 0);
    const int x = x0 + r, yq = y0 + 4 * q;
    const bool row_ok = r < tile_x && x < nx - kRadius;
    unsigned okb = 0, fyb = 0;   // bits per cell: updated; of a y face
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        const int y = yq + j;
        if (row_ok && y >= kRadius && y < ny - kRadius) okb |= 1u << j;
        if (y < pml || y >= ny - pml) fyb |= 1u << j;
    }
    const bool mem_ok = okb != 0, y_inner = yq >= pml && yq + 3 < ny - pml;
    const int fx = x < pml ? 0 : (x >= nx - pml ? 1 : -1);
    const int lix = x < pml ? pml - x : x - nx + pml;
    const bool xy_face = row_ok && (fx >= 0 || (fyb & okb));
    const bool xy_face_warp = __any_sync(0xffffffffu, xy_face);
    auto face_of_z = [&](int z) { return z < pml ? 4 : (z >= nz - pml ? 5 : -1); };
    float4 *own = reinterpret_cast<float4 *>(smem + L.own_off) + tid;
    const int nthr = blockDim.x;
    unsigned base = (unsigned)((long long)z0 * a.plane + (long long)x * a.ldy + yq);
    const unsigned plane = (unsigned)a.plane;
    auto prefetch_params = [&](unsigned b) {
        if (!mem_ok) return;
        cp_async16(own + 2 * nthr, a.VP + b);
        cp_async16(own + 3 * nthr, a.E2 + b);
        cp_async16(own + 4 * nthr, a.R8 + b);
    };
    auto prefetch = [&](unsigned b, int z) {
        if (!mem_ok) return;
        cp_async16(own, a.Lu + b);
        cp_async16(own + nthr, a.Lprev + b);
        const bool z_face = face_of_z(z) >= 0;
        if (!(fx >= 0 || z_face || (fyb & okb) == okb)) {   // a cell of the interior
            cp_async16(own + 5 * nthr, a.gK + b);
            cp_async16(own + 6 * nthr, a.gE + b);
            cp_async16(own + 7 * nthr, a.gD + b);
        }
        if (xy_face || z_face) {
            cp_async16(own + 8 * nthr, a.Lw1 + b);
            cp_async16(own + 9 * nthr, a.Lw21 + b);
            cp_async16(own + 10 * nthr, a.Lw3 + b);
            cp_async16(own + 11 * nthr, a.Lp + b);
            cp_async16(own + 12 * nthr, a.Lw1o + b);
            cp_async16(own + 13 * nthr, a.Lpo + b);
            cp_async16(own + 14 * nthr, a.Lw3o + b);
        }
    };
    prefetch_params(base);
    if (tid == 0) pipe_init(P);
    for (int i = tid; i < 3 * pml; i += blockDim.x) tab[i] = fast_layer(a.layers[i]);
    pdl_wait();
    if (tid == 0) pipe_start(P, &tm);
    prefetch(base, z0);
    const float T2 = *a.T2;
    __syncthreads();
    const Coefs &k = a.k;
    Taps T = taps_start(P, r, q);
    bool ok = true;
    auto plane_adj = [&](int t, auto shell) {
        constexpr bool PML = decltype(shell)::value;
        const int z = z0 + t;
        const int fz = PML ? face_of_z(z) : -1;
        cp_async_wait();
        const float4 lu = own[0], lq = own[nthr], Vv = own[2 * nthr], Ev = own[3 * nthr],
                     Rv = own[4 * nthr], vK = own[5 * nthr], vE = own[6 * nthr],
                     vD = own[7 * nthr];
        float4 vw1, vw21, vw3, vp, vw1o, vpo, vw3o;
        const bool pml_quad = PML && (xy_face || (row_ok && fz >= 0));
        if (pml_quad) {
            vw1 = own[8 * nthr]; vw21 = own[9 * nthr]; vw3 = own[10 * nthr]; vp = own[11 * nthr];
            vw1o = own[12 * nthr]; vpo = own[13 * nthr]; vw3o = own[14 * nthr];
        }
        if (t + 1 < nzc) {
            prefetch(base + plane, z + 1);
            prefetch_params(base + plane);
        }
        ok = __all_sync(0xffffffffu, pipe_wait(P, t));
        if (!ok) return;
        float Ux[4], Uy[4], Uz[4], Uxx[4], Uyy[4], Uzz[4];
        adj_derivs(T, k, Ux, Uy, Uz, Uxx, Uyy, Uzz);
        // the adjoint of u, and that of the step after: the residual is added
        // at the receivers
        float l[4] = {lu.x, lu.y, lu.z, lu.w}, lp[4] = {lq.x, lq.y, lq.z, lq.w};
        if (z == a.sz && row_ok && x >= pml && x < nx - pml) {
#pragma unroll
            for (int j = 0; j < 4; ++j)
                if (yq + j >= pml && yq + j < ny - pml) {
                    const long long i = (long long)(x - pml) * a.hy + (yq + j - pml);
                    l[j] += a.resid[i];
                    if (a.resid_prev) lp[j] += a.resid_prev[i];
                }
        }
        float nu[4] = {0.f, 0.f, 0.f, 0.f};
        // frozen scalar operator and its eps / delta derivatives
        const float4 Kv = make_float4(k_of_vp(Vv.x, a.dt), k_of_vp(Vv.y, a.dt),
                                      k_of_vp(Vv.z, a.dt), k_of_vp(Vv.w, a.dt));
        // wa: with the live operator, dS/da times 2 / m2, so that the
        // derivatives of S in Ux, Uy, Uz are wa (Ux (1 - a), Uy (1 - a), -Uz a)
        // (a = h2 / m2 = nx^2 + ny^2, h2 = Ux^2 + Uy^2, m2 = h2 + Uz^2; no
        // power of m2 above the first, which could leave the float range)
        float KS[4], e2[4], S[4], dSe[4], dSd[4], wa[4], av[4], m2[4], h2[4];
        unsigned on = 0;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            h2[j] = fmaf(Uy[j], Uy[j], Ux[j] * Ux[j]);
            m2[j] = fmaf(Uz[j], Uz[j], h2[j]);
            if (m2[j] > T2) on |= 1u << j;
            S[j] = 1.0f;
            dSe[j] = dSd[j] = wa[j] = av[j] = 0.0f;
            e2[j] = 1.0f + f4(Ev, j);
        }
        if (a.dec && row_ok) on = (a.dec[base >> 5] >> (4 * q)) & 15u;
        if (__any_sync(0xffffffffu, on & okb)) {
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const float E2 = f4(Ev, j), R8 = f4(Rv, j);
                const float aa = __fdividef(h2[j], m2[j]), bb = 1.0f - aa, D = fmaf(E2, aa, 1.0f);
                const float iD = __fdividef(1.0f, D);
                const float ab8 = 8.0f * aa * bb * iD * iD;
                const float qq = 0.125f * R8 * ab8;
                const float rr = sqrtf(fmaxf(1.0f - qq, 0.0f));
                const float dSdq = rr > 0.0f ? __fdividef(-0.25f, rr) : 0.0f;
                // dq/da = R8 ((1 - 2a) D - 2 E2 a (1 - a)) / D^3
                const float dqda = R8 * ((1.0f - 2.0f * aa) * D - 2.0f * E2 * aa * bb) * iD * iD * iD;
                if (on >> j & 1u) {
                    S[j] = 0.5f + 0.5f * rr;
                    dSe[j] = dSdq * ab8 * (1.0f - 0.5f * aa * R8 * iD);
                    dSd[j] = -dSdq * ab8;
                    if (a.live) {
                        wa[j] = __fdividef(2.0f * dSdq * dqda, m2[j]);
                        av[j] = aa;
                    }
                }
            }
        }
#pragma unroll
        for (int j = 0; j < 4; ++j) KS[j] = f4(Kv, j) * S[j];
        float c0[4], c1[4], c2[4], c3[4], c4[4], c5[4];
        const unsigned pmlb = PML ? (fx >= 0 || fz >= 0 ? 15u : fyb) & okb : 0u;
        const unsigned intb = okb & ~pmlb;
        if (PML) {
#pragma unroll
            for (int j = 0; j < 4; ++j) c0[j] = c1[j] = c2[j] = c3[j] = c4[j] = c5[j] = 0.0f;
        }
        if (!PML || intb) {   // interior leapfrog and the gradient sums
            float gK[4] = {vK.x, vK.y, vK.z, vK.w}, gE[4] = {vE.x, vE.y, vE.z, vE.w},
                  gD[4] = {vD.x, vD.y, vD.z, vD.w};
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const bool in = (intb >> j) & 1u;
                // u_prev's adjoint is -l of the step after (0 in the shell)
                const float n2 = -lp[j] + 2.0f * l[j];
                const float cc = KS[j] * e2[j] * l[j];
                const float Lh = Uxx[j] + Uyy[j], Lap = fmaf(e2[j], Lh, Uzz[j]);
                const float Kc = f4(Kv, j);
                const float aK = gK[j] + l[j] * S[j] * Lap;
                const float aE = gE[j] + l[j] * Kc * (2.0f * S[j] * Lh + dSe[j] * Lap);
                const float aD = gD[j] + l[j] * Kc * dSd[j] * Lap;
                // live operator: S's dependence on grad u, through the
                // transposed first derivatives (zero where S = 1)
                const float w = l[j] * Kc * Lap * wa[j], bv = 1.0f - av[j];
                if (in) {
                    nu[j] = n2;
                    c3[j] = c4[j] = cc;
                    c5[j] = KS[j] * l[j];
                    gK[j] = aK; gE[j] = aE; gD[j] = aD;
                    c0[j] = w * Ux[j] * bv;
                    c1[j] = w * Uy[j] * bv;
                    c2[j] = -w * Uz[j] * av[j];
                } else if (!PML) {
                    gK[j] = gE[j] = gD[j] = 0.0f;
                    c0[j] = c1[j] = c2[j] = c3[j] = c4[j] = c5[j] = 0.0f;
                }
            }
            if (mem_ok) {
                QP3D_ST4(a.gK, gK); QP3D_ST4(a.gE, gE); QP3D_ST4(a.gD, gD);
            }
        }
        if (PML && pml_quad) {   // transposed split-field recursions
            float nw1[4], nw1o[4], np_[4], npo[4], nw21[4], nw3[4], nw3o[4];
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                nw1[j] = nw1o[j] = np_[j] = npo[j] = nw21[j] = nw3[j] = nw3o[j] = 0.0f;
                if (!((pmlb >> j) & 1u)) continue;
                int f, li;
                const int y = yq + j;
                const int fy = y < pml ? 2 : (y >= ny - pml ? 3 : -1);
                cell_face(fx, lix, fy, y < pml ? pml - y : y - ny + pml, fz,
                          z < pml ? pml - z : z - nz + pml, f, li);
                const float4 lc = tab[(f >> 1) * pml + li];
                const bool isz = f >= 4;
                const float A = isz ? KS[j] : e2[j] * KS[j], Bt = isz ? e2[j] * KS[j] : KS[j];
                const float sgn = (f & 1) ? -1.0f : 1.0f;
                const float W1 = f4(vw1, j) + l[j], W21 = f4(vw21, j) + l[j], W3 = f4(vw3, j) + l[j];
                const float Pp = fmaf(a.dt, W21, f4(vp, j));
                nw1[j] = fmaf(-lc.x, W1, f4(vw1o, j));
                nw1o[j] = lc.y * W1;
                np_[j] = fmaf(-lc.x, Pp, f4(vpo, j));
                npo[j] = lc.y * Pp;
                nw21[j] = lc.z * W21;
                nw3[j] = fmaf(2.0f, W3, f4(vw3o, j));
                nw3o[j] = -W3;
                const float cn = A * W1, cf = sgn * A * lc.w * Pp, ct = Bt * W3;
                if (f < 2) { c3[j] = cn; c0[j] = cf; c4[j] = ct * e2[j]; c5[j] = ct; }
                else if (f < 4) { c4[j] = cn; c1[j] = cf; c3[j] = ct * e2[j]; c5[j] = ct; }
                else { c5[j] = cn; c2[j] = cf; c3[j] = ct; c4[j] = ct; }
                if (a.live && wa[j] != 0.0f) {
                    // the S-proportional terms of w1', p' and w3' (their
                    // weights cn, cf, ct over S) times dS/d(grad u)
                    const float Unn = f < 2 ? Uxx[j] : (isz ? Uzz[j] : Uyy[j]);
                    const float Un = f < 2 ? Ux[j] : (isz ? Uz[j] : Uy[j]);
                    const float tang = isz ? Uxx[j] + Uyy[j]
                                           : fmaf(e2[j], f < 2 ? Uyy[j] : Uxx[j], Uzz[j]);
                    const float w = __fdividef(cn * Unn + cf * Un + ct * tang, S[j]) * wa[j];
                    const float bv = 1.0f - av[j];
                    c0[j] += w * Ux[j] * bv;
                    c1[j] += w * Uy[j] * bv;
                    c2[j] -= w * Uz[j] * av[j];
                }
            }
            if (mem_ok) {
                QP3D_ST4(a.Nw1, nw1); QP3D_ST4(a.Nw1o, nw1o); QP3D_ST4(a.Np, np_);
                QP3D_ST4(a.Npo, npo); QP3D_ST4(a.Nw21, nw21); QP3D_ST4(a.Nw3, nw3);
                QP3D_ST4(a.Nw3o, nw3o);
            }
        }
        if (mem_ok) {
            if (pml_quad || a.live) {
                QP3D_ST4(a.C[0], c0); QP3D_ST4(a.C[1], c1); QP3D_ST4(a.C[2], c2);
            }
            QP3D_ST4(a.C[3], c3); QP3D_ST4(a.C[5], c5);
            // Cyy equals Cxx at cells of the interior: pass B takes it from there
            // for quads that hold nothing else
            if (!y_inner || (PML && pml_quad)) QP3D_ST4(a.C[4], c4);
            QP3D_ST4(a.Nu, nu);
        }
        pipe_release(P, &tm, t);
    };
    for (int t = 0; t < nzc && ok; taps_next(T, P, t), ++t, base += plane) {
        if (xy_face_warp || face_of_z(z0 + t) >= 0) plane_adj(t, std::true_type());
        else plane_adj(t, std::false_type());
    }
    cp_async_wait();
    pipe_finish(P, ok, a.err);
}
#undef QP3D_ST4

// Pass B: Nu += the transposed stencils of the six coefficient fields, over
// the updated cells (their taps lie inside the volume; along y the rows are
// padded to whole quads, and taps before a row's start or past its end read
// zero).  Bound by the latency of its 53 16-byte loads a quad through L1:
// 240x240x190 105 us with every cell of the volume, 89 with the updated cells
// in 44 registers.
__device__ __forceinline__ void fma4(float acc[4], float c, const float4 &a, const float4 &b, bool minus)
{
#pragma unroll
    for (int j = 0; j < 4; ++j)
        acc[j] = fmaf(c, minus ? f4(a, j) - f4(b, j) : f4(a, j) + f4(b, j), acc[j]);
}

// A thread takes one quad.  With the frozen operator, a warp whose whole
// footprint (its cells and 5 around them) lies outside the shell, where Cx, Cy,
// Cz are zero and Cyy equals Cxx (qp3d_adj_a_kernel), reads two fields.
// Two rows by two planes of quads per thread, which needs 34 16-byte loads a
// quad instead of 53, left 16 warps an SM and took 111 us instead of 105 on
// 240x240x190: the pass waits for latency rather than for the bytes.  Marching
// along z with the planes of Cz and Czz in registers (33 loads a quad, 168
// registers, 12 warps an SM) took 117 against 89 us; CTAs of 16 rows by 2 planes
// 92, 8 by 4 95, 4 by 8 104, although they halve what misses L1.
__global__ void __launch_bounds__(256) qp3d_adj_b_kernel(const AdjParams a)
{
    pdl_trigger();
    pdl_wait();
    const int q = threadIdx.x & 7, r = threadIdx.x >> 3;
    const int y = blockIdx.x * 32 + 4 * q, x = blockIdx.y * 32 + r;
    const int z = kRadius + blockIdx.z;
    if (y + 3 < kRadius || y >= a.ny - kRadius || x < kRadius || x >= a.nx - kRadius) return;
    const int xw = blockIdx.y * 32 + ((threadIdx.x >> 5) << 2), yw = blockIdx.x * 32;
    const long long i = (long long)z * a.plane + (long long)x * a.ldy + y;
    const Coefs &k = a.k;
    // the quad's Nu, read-modified-written at the end, moves to shared memory
    // while the taps are gathered (7% of the pass on a 240x240x190 grid)
    __shared__ __align__(16) float4 pnu[256];
    cp_async16(&pnu[threadIdx.x], a.Nu + i);
    const bool inside = !a.live && xw - kRadius >= a.pml && xw + 4 + kRadius <= a.nx - a.pml &&
                        yw - kRadius >= a.pml && yw + 32 + kRadius <= a.ny - a.pml &&
                        z - kRadius >= a.pml && z + kRadius < a.nz - a.pml;
    float acc[4];
    const float *Cx = a.C[0], *Cy = a.C[1], *Cz = a.C[2], *Cxx = a.C[3], *Cyy = a.C[4],
                *Czz = a.C[5];
    float w[20];
    // Cyy, of quads wholly in the interior kept in Cxx only
    const bool row_in = x >= a.pml && x < a.nx - a.pml && z >= a.pml && z < a.nz - a.pml;
#pragma unroll
    for (int b = 0; b < 5; ++b) {
        const int yb = y - 8 + 4 * b;
        const bool in = row_in && yb >= a.pml && yb + 3 < a.ny - a.pml;
        const float4 v = ldg4_or0(in ? Cxx : Cyy, i - 8 + 4 * b, yb >= 0 && yb < a.ldy);
        w[4 * b] = v.x; w[4 * b + 1] = v.y; w[4 * b + 2] = v.z; w[4 * b + 3] = v.w;
    }
    const float4 xx0 = ldg4_or0(Cxx, i, true), zz0 = ldg4_or0(Czz, i, true);
#pragma unroll
    for (int j = 0; j < 4; ++j) acc[j] = k.kx * f4(xx0, j) + k.ky * w[8 + j] + k.kz * f4(zz0, j);
    if (inside) {
#pragma unroll
        for (int m = 0; m < kRadius; ++m) {
            const int d = m + 1;
            const long long dx = (long long)d * a.ldy, dz = (long long)d * a.plane;
            fma4(acc, k.c2x[m], ldg4_or0(Cxx, i + dx, true), ldg4_or0(Cxx, i - dx, true), false);
#pragma unroll
            for (int j = 0; j < 4; ++j) acc[j] = fmaf(k.c2y[m], w[8 + j + d] + w[8 + j - d], acc[j]);
            fma4(acc, k.c2z[m], ldg4_or0(Czz, i + dz, true), ldg4_or0(Czz, i - dz, true), false);
        }
    } else {
#pragma unroll
        for (int m = 0; m < kRadius; ++m)
#pragma unroll
            for (int j = 0; j < 4; ++j)
                acc[j] = fmaf(k.c2y[m], w[8 + j + m + 1] + w[8 + j - m - 1], acc[j]);
        row_window(Cy, i, y, a.ldy, w);
#pragma unroll
        for (int m = 0; m < kRadius; ++m)
#pragma unroll
            for (int j = 0; j < 4; ++j)
                acc[j] = fmaf(k.cy[m], w[8 + j - m - 1] - w[8 + j + m + 1], acc[j]);
#pragma unroll
        for (int m = 0; m < kRadius; ++m) {
            const int d = m + 1;
            const long long dx = (long long)d * a.ldy, dz = (long long)d * a.plane;
            fma4(acc, k.c2x[m], ldg4_or0(Cxx, i + dx, true), ldg4_or0(Cxx, i - dx, true), false);
            fma4(acc, k.c2z[m], ldg4_or0(Czz, i + dz, true), ldg4_or0(Czz, i - dz, true), false);
            fma4(acc, k.cx[m], ldg4_or0(Cx, i - dx, true), ldg4_or0(Cx, i + dx, true), true);
            fma4(acc, k.cz[m], ldg4_or0(Cz, i - dz, true), ldg4_or0(Cz, i + dz, true), true);
        }
    }
    cp_async_wait();
    float4 v = pnu[threadIdx.x];
    v.x += acc[0]; v.y += acc[1]; v.z += acc[2]; v.w += acc[3];
    *reinterpret_cast<float4 *>(a.Nu + i) = v;
}

__global__ void qp3d_threshold_kernel(const float *gmax, float *T2, int n)
{
    for (int i = threadIdx.x; i < n; i += blockDim.x) T2[i] = threshold_m2(gmax[i]);
}

// Record residual r = record - d_obs and the misfit 1/2 sum r^2 (FP64, one
// atomic per block).
__global__ void qp3d_residual_kernel(const float *rec, const float *dobs, float *r, long long n,
                                     double *misfit)
{
    __shared__ double s[32];
    double acc = 0.0;
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n;
         i += (long long)gridDim.x * blockDim.x) {
        const float v = rec[i] - dobs[i];
        r[i] = v;
        acc += 0.5 * (double)v * (double)v;
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
    if ((threadIdx.x & 31) == 0) s[threadIdx.x >> 5] = acc;
    __syncthreads();
    if (threadIdx.x == 0) {
        double t = 0.0;
        for (int w = 0; w < (int)(blockDim.x >> 5); ++w) t += s[w];
        atomicAdd(misfit, t);
    }
}

__global__ void qp3d_to_bf16_kernel(const float *a, __nv_bfloat16 *h, long long n)
{
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n;
         i += (long long)gridDim.x * blockDim.x)
        h[i] = __float2bfloat16_rn(a[i]);
}

__global__ void qp3d_from_bf16_kernel(const __nv_bfloat16 *h, float *a, long long n)
{
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n;
         i += (long long)gridDim.x * blockDim.x)
        a[i] = __bfloat162float(h[i]);
}

// ---------------------------------------------------------------------------
// Launchers
// ---------------------------------------------------------------------------
// A kernel of a time step, as a programmatic dependent of the one before it.
template <typename... P, typename... A>
static cudaError_t launch_pdl(void (*fn)(P...), dim3 grid, int threads, size_t smem,
                              cudaStream_t stream, const A &...args)
{
    cudaLaunchAttribute at;
    at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t c = {};
    c.gridDim = grid;
    c.blockDim = dim3(threads);
    c.dynamicSmemBytes = smem;
    c.stream = stream;
    c.attrs = &at;
    c.numAttrs = 1;
    return cudaLaunchKernelEx(&c, fn, args...);
}

template <typename F>
static cudaError_t set_smem(F *fn, int bytes)
{
    return cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
}

cudaError_t configure_kernels()
{
    const int bytes = 200 * 1024;
    cudaError_t e;
    if ((e = set_smem(qp3d_batch_plane_kernel<0, kArithFast>, bytes)) ||
        (e = set_smem(qp3d_batch_plane_kernel<1, kArithFast>, bytes)) ||
        (e = set_smem(qp3d_batch_plane_kernel<2, kArithFast>, bytes)) ||
        (e = set_smem(qp3d_batch_plane_kernel<0, kArithRef>, bytes)) ||
        (e = set_smem(qp3d_batch_plane_kernel<1, kArithRef>, bytes)) ||
        (e = set_smem(qp3d_batch_plane_kernel<2, kArithRef>, bytes)) ||
        (e = set_smem(qp3d_batch_resolve_kernel<kArithFast>, bytes)) ||
        (e = set_smem(qp3d_adj_a_kernel, bytes)) ||
        (e = set_smem(qp3d_batch_resolve_kernel<kArithRef>, bytes)))
        return e;
#define QP3D_STEP_SMEM(AR)                                                                   \
    if ((e = set_smem(qp3d_step_kernel<true, false, AR>, bytes)) ||                         \
        (e = set_smem(qp3d_step_kernel<false, false, AR>, bytes)) ||                        \
        (e = set_smem(qp3d_step_kernel<true, false, AR, true>, bytes)) ||                   \
        (e = set_smem(qp3d_step_kernel<true, true, AR>, bytes)) ||                          \
        (e = set_smem(qp3d_step_kernel<false, true, AR>, bytes)) ||                         \
        (e = set_smem(qp3d_gradmax_kernel<AR>, bytes)) ||                                   \
        (e = set_smem(qp3d_fix_or_rerun_kernel<false, AR>, bytes)) ||                              \
        (e = set_smem(qp3d_fix_or_rerun_kernel<true, AR>, bytes)))                                 \
        return e;
    QP3D_STEP_SMEM(kArithFast)
    QP3D_STEP_SMEM(kArithRef)
#undef QP3D_STEP_SMEM
    return cudaSuccess;
}

cudaError_t launch_gradmax(const TileMaps &tm, const PlaneParams &p, dim3 grid,
                           cudaStream_t stream)
{
    const int t = plane_threads(p.tile_x);
    const size_t smem = gradmax_smem_bytes(p.tile_x);
    return launch_pdl(p.arith == kArithRef ? qp3d_gradmax_kernel<kArithRef>
                                           : qp3d_gradmax_kernel<kArithFast>,
                      grid, t, smem, stream, tm, p);
}

template <int AR>
static cudaError_t launch_step_t(const TileMaps &tm, const PlaneParams &p, dim3 grid, int t,
                                 size_t smem, cudaStream_t stream)
{
    auto *fn = p.half_params ? (p.spec ? qp3d_step_kernel<true, true, AR>
                                       : qp3d_step_kernel<false, true, AR>)   // no decisions kept
               : !p.spec     ? qp3d_step_kernel<false, false, AR>
               : p.dec_out   ? qp3d_step_kernel<true, false, AR, true>
                             : qp3d_step_kernel<true, false, AR>;
    return launch_pdl(fn, grid, t, smem, stream, tm, p);
}

cudaError_t launch_step(const TileMaps &tm, const PlaneParams &p, dim3 grid, size_t smem,
                        cudaStream_t stream)
{
    const int t = plane_threads(p.tile_x);
    return p.arith == kArithRef ? launch_step_t<kArithRef>(tm, p, grid, t, smem, stream)
                                : launch_step_t<kArithFast>(tm, p, grid, t, smem, stream);
}

cudaError_t configure_gradmax_single()
{
    return set_smem(qp3d_gradmax_single_kernel, 200 * 1024);
}

cudaError_t launch_gradmax_direct(const float *u, int nx, int ny, int nz, int ldy, const Coefs &k,
                                  int nsm, cudaStream_t stream, GradmaxScratch *sc, float *out,
                                  unsigned *host_flags)
{
    const int rows = kDirectThreads / 8, ncz = nz - 2 * kRadius;
    const unsigned nyt = (ny - kRadius - 1) / kTileY + 1;
    const unsigned nxt = (nx - 2 * kRadius + rows - 1) / rows;
    const int n = plan_chunks((long long)nyt * nxt, ncz, kDirectThreads, 0, nsm);
    const int chunk = (ncz + n - 1) / n;
    const unsigned nch = (ncz + chunk - 1) / chunk;
    qp3d_gradmax_direct_kernel<<<dim3(nyt, nxt, nch), kDirectThreads, 0, stream>>>(
        u, nx, ny, nz, ldy, chunk, k, sc, out, host_flags);
    return cudaGetLastError();
}

cudaError_t launch_gradmax_single(const TileMaps &tm, const PlaneParams &p, dim3 grid,
                                  cudaStream_t stream, GradmaxScratch *sc, float *out,
                                  unsigned *host_flags)
{
    qp3d_gradmax_single_kernel<<<grid, plane_threads(p.tile_x), gradmax_smem_bytes(p.tile_x),
                                 stream>>>(tm, p, sc, out, host_flags);
    return cudaGetLastError();
}

template <int AR>
static cudaError_t launch_fix_or_rerun_t(const TileMaps &tm, const PlaneParams &p,
                                         float *spec_err, int grid, int t, size_t smem,
                                         cudaStream_t stream)
{
    return launch_pdl(p.half_params ? qp3d_fix_or_rerun_kernel<true, AR>
                                    : qp3d_fix_or_rerun_kernel<false, AR>,
                      dim3(grid), t, smem, stream, tm, p, spec_err);
}

cudaError_t launch_fix_or_rerun(const TileMaps &tm, const PlaneParams &p, float *spec_err,
                                int nsm, size_t smem, cudaStream_t stream)
{
    const int t = plane_threads(p.tile_x);
    return p.arith == kArithRef
               ? launch_fix_or_rerun_t<kArithRef>(tm, p, spec_err, 2 * nsm, t, smem, stream)
               : launch_fix_or_rerun_t<kArithFast>(tm, p, spec_err, 2 * nsm, t, smem, stream);
}

cudaError_t launch_batch_prepare(const BatchShot *shots, int nshots, PlaneParams *pp, int *ctr,
                                 int *queue, int spec, cudaStream_t stream)
{
    return launch_pdl(qp3d_batch_prepare_kernel, dim3(1), 128, 0, stream, shots, nshots, pp, ctr,
                      queue, spec);
}

template <int AR>
static cudaError_t launch_batch_plane_t(int kind, const BatchArgs &b, int threads, size_t smem,
                                        cudaStream_t stream)
{
    auto *fn = kind == 0 ? qp3d_batch_plane_kernel<0, AR>
             : kind == 1 ? qp3d_batch_plane_kernel<1, AR> : qp3d_batch_plane_kernel<2, AR>;
    return launch_pdl(fn, dim3(b.nwork), threads, smem, stream, b);
}

cudaError_t launch_batch_plane(int kind, const BatchArgs &b, int threads, size_t smem,
                               cudaStream_t stream)
{
    return b.arith == kArithRef ? launch_batch_plane_t<kArithRef>(kind, b, threads, smem, stream)
                                : launch_batch_plane_t<kArithFast>(kind, b, threads, smem, stream);
}

cudaError_t launch_batch_resolve(const BatchArgs &b, int grid, int threads, size_t smem,
                                 cudaStream_t stream)
{
    return launch_pdl(b.arith == kArithRef ? qp3d_batch_resolve_kernel<kArithRef>
                                           : qp3d_batch_resolve_kernel<kArithFast>,
                      dim3(grid), threads, smem, stream, b);
}

cudaError_t launch_band_sources(float *u_new, const float *u_cur, const SrcEntry *src, int n,
                                long long plane, int ldy, float w, cudaStream_t stream)
{
    if (n <= 0) return cudaSuccess;
    qp3d_band_source_kernel<<<(n + 127) / 128, 128, 0, stream>>>(u_new, u_cur, src, n, plane, ldy,
                                                                 w);
    return cudaGetLastError();
}

cudaError_t launch_all_sources(float *u_new, const float *u_cur, const SrcEntry *src, int n,
                               long long plane, int ldy, int nx, int ny, int nz, float w,
                               cudaStream_t stream)
{
    if (n <= 0) return cudaSuccess;
    qp3d_all_source_kernel<<<(n + 255) / 256, 256, 0, stream>>>(u_new, u_cur, src, n, plane, ldy,
                                                                nx, ny, nz, w);
    return cudaGetLastError();
}

cudaError_t launch_record(const float *u, float *rec, int nx, int ny, int pml, int sz, int ldy,
                          long long plane, cudaStream_t stream)
{
    long long n = (long long)(nx - 2 * pml) * (ny - 2 * pml);
    int blocks = (int)((n + 255) / 256);
    if (blocks > 4096) blocks = 4096;
    if (blocks < 1) blocks = 1;
    qp3d_record_kernel<<<blocks, 256, 0, stream>>>(u, rec, nx, ny, pml, sz, ldy, plane);
    return cudaGetLastError();
}

cudaError_t launch_crop(const float *u, float *out, int x0, int x1, int y0, int y1, int z0, int z1,
                        int ldy, long long plane, cudaStream_t stream)
{
    long long n = (long long)(x1 - x0) * (y1 - y0) * (z1 - z0);
    if (n <= 0) return cudaSuccess;
    long long b = (n + 255) / 256;
    int blocks = (int)(b > 8192 ? 8192 : b);
    qp3d_crop_kernel<<<blocks, 256, 0, stream>>>(u, out, x0, x1, y0, y1, z0, z1, ldy, plane);
    return cudaGetLastError();
}

void plan_adjoint(AdjParams &a, int nsm)
{
    const int ncx = a.nx - 2 * kRadius, ncz = a.nz - 2 * kRadius;
    const int ntx = (ncx + kAdjTileX - 1) / kAdjTileX;
    a.tile_x = (ncx + ntx - 1) / ntx;
    const long long tiles = (long long)ntx * ((a.ny - kRadius - 1) / kTileY + 1);
    const size_t smem = smem_layout(a.tile_x, a.pml, 0, kAdjStreams).total;
    // Where there are several waves either way, short chunks keep more loads
    // and stores in flight: 5 planes 189 us on 240x240x190, 12 planes (the
    // estimate's choice) 199.  On either side of the line, whole gradients of 120
    // steps with 5 planes and with the estimate's: 300x300x200 (32 CTAs an SM)
    // 80.7 and 83.4 ms, 240x240x190 (19) 54.3 and 56.0; below it, where the
    // estimate is taken, 200x200x150 (10) 33.1 and 36.0, 150x150x150 (5.5) 20.9
    // and 22.5, 130x130x110 (2.6) 13.4 and 12.8, 100x100x100 (1.4) 9.0 and 8.5: the
    // crossover is near 4, and the line could lie there.
    const int n = tiles * ((ncz + 4) / 5) >= 12ll * nsm
                      ? (ncz + 4) / 5
                      : plan_chunks(tiles, ncz, std::max(192, plane_threads(a.tile_x)), smem, nsm);
    a.chunk_z = (ncz + n - 1) / n;
}

cudaError_t launch_adjoint_step(const TileMaps &tm, const AdjParams &a, cudaStream_t stream)
{
    const int nyt = (a.ny - kRadius - 1) / kTileY + 1;
    const int nxt = (a.nx - 2 * kRadius + a.tile_x - 1) / a.tile_x;
    const int nch = (a.nz - 2 * kRadius + a.chunk_z - 1) / a.chunk_z;
    cudaError_t e = launch_pdl(qp3d_adj_a_kernel, dim3(nyt, nxt, nch), plane_threads(a.tile_x),
                               smem_layout(a.tile_x, a.pml, 0, kAdjStreams).total, stream, tm, a);
    if (e != cudaSuccess) return e;
    const int ncz = a.nz - 2 * kRadius;
    return launch_pdl(qp3d_adj_b_kernel, dim3(nyt, (a.nx + 31) / 32, ncz), 256, 0,
                      stream, a);
}

cudaError_t launch_threshold(const float *gmax, float *T2, int n, cudaStream_t stream)
{
    qp3d_threshold_kernel<<<1, 256, 0, stream>>>(gmax, T2, n);
    return cudaGetLastError();
}

cudaError_t launch_residual(const float *rec, const float *dobs, float *r, long long n,
                            double *misfit, cudaStream_t stream)
{
    if (n <= 0) return cudaSuccess;
    long long b = (n + 255) / 256;
    qp3d_residual_kernel<<<(int)(b > 4096 ? 4096 : b), 256, 0, stream>>>(rec, dobs, r, n, misfit);
    return cudaGetLastError();
}

cudaError_t launch_to_bf16(const float *a, __nv_bfloat16 *h, long long n, cudaStream_t stream)
{
    if (n <= 0) return cudaSuccess;
    long long b = (n + 255) / 256;
    qp3d_to_bf16_kernel<<<(int)(b > 8192 ? 8192 : b), 256, 0, stream>>>(a, h, n);
    return cudaGetLastError();
}

cudaError_t launch_from_bf16(const __nv_bfloat16 *h, float *a, long long n, cudaStream_t stream)
{
    if (n <= 0) return cudaSuccess;
    long long b = (n + 255) / 256;
    qp3d_from_bf16_kernel<<<(int)(b > 8192 ? 8192 : b), 256, 0, stream>>>(h, a, n);
    return cudaGetLastError();
}

cudaError_t launch_params_dense(const float *vp, const float *eps, const float *del, float *VP,
                                float *E2, float *R8, int nx, int ny, int nz, int ldy,
                                cudaStream_t stream)
{
    const long long vol = (long long)nz * nx * ldy;
    const long long b = (vol + 255) / 256;
    qp3d_params_dense_kernel<<<(int)(b > 16384 ? 16384 : b), 256, 0, stream>>>(
        vp, eps, del, VP, E2, R8, ny, vol, ldy);
    return cudaGetLastError();
}

cudaError_t launch_to_half_dense(const float *a, __half *h, int nx, int ny, int nz, int ldy,
                                 cudaStream_t stream)
{
    const long long vol = (long long)nz * nx * ldy;
    const long long b = (vol + 255) / 256;
    qp3d_to_half_dense_kernel<<<(int)(b > 16384 ? 16384 : b), 256, 0, stream>>>(a, h, ny, vol,
                                                                                ldy);
    return cudaGetLastError();
}

}  // namespace qp3d
