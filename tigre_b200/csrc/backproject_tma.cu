// Voxel-driven backprojection with TMA-staged projection patches (sm_100a).
//
// Same arithmetic as backproject.cu (FDK weight of voxel_backprojection.cu:242-249,
// matched weight of voxel_backprojection2.cu:256-280, bilinear sampling with border 0),
// organised for the B200 memory system:
//
//  * a block owns 16 x 16 voxel columns x 64 slices (one thread per column,
//    64 accumulators in registers; a warp covers 8 x 4 columns) and loops over
//    every view of the call, so the volume is written once per call;
//  * for each view, the bilinear footprint of the block's voxels lies inside
//    the bounding box of its 8 projected corners; one elected lane issues a
//    cp.async.bulk.tensor load of that box of the projection into shared
//    memory (TMA zero-fills what lies outside the detector, which is exactly
//    the texture border rule), double-buffered on two mbarriers so the next
//    view's patch streams in while the current one is consumed;
//  * all per-view constants are precomputed on the host (FrameBPK), so a
//    (column, view) costs a few FP64 FMAs and one division, and a voxel
//    update a handful of packed FP32x2 instructions and four shared-memory
//    loads; the matched weight along a column is a cubic fitted at four
//    Chebyshev nodes per (column, view);
//  * every mbarrier wait is bounded, and a thread whose wait expired waits no
//    more; warp 0's lane 0 issues a copy into a buffer only while its own
//    waits have all succeeded (so only into a buffer whose previous copy has
//    landed); the warps of a thread that saw an expiry write nothing and set
//    TIGRE_STATUS_WAIT_EXPIRED in the plan's status word, and thread 0 waits,
//    bounded, for the copies it issued that may still be in flight -- the
//    block ends instead of hanging.  The steady state carries no extra block
//    barrier or shared flag for this (measured: either costs 2-3 %).
// A (block, view) whose footprint does not fit the box (possible for strongly
// magnified geometries) falls back to bounds-checked global loads.
//
// Small volumes give few blocks (64^3: 16 for 148 SMs), each serially over all views, so the
// views of a tile are then divided over a cluster of 2, 4 or 8 blocks (bp_splits): every block
// sums its share of the views in registers as above, leaves the sums in shared memory, and each
// adds up and writes its part of the tile's slices through distributed shared memory, in
// a fixed order.  No workspace, no second launch, one rounding to the storage type.

#include <type_traits>
#include <cooperative_groups.h>
#include <cuda.h>
#include <cudaTypedefs.h>

#include <cmath>
#include <mutex>

#include "tigre_internal.h"

namespace tigre {
namespace {

constexpr int TXY = kBpTile;   // columns per block edge
constexpr int VZ = kBpSlices;  // slices per thread
constexpr int kMaxSplit = 8;   // blocks per tile at most: the portable cluster size
constexpr unsigned kWaitLimit = 1u << 16;   // ~ a few ms with the back-off below

struct BPKArgs {
    const FrameBPK* frames;
    const void* proj;     // projection buffer the tensor map describes (fallback reads)
    void* vol;
    int* status;
    int a0, na;
    int nX, nY, nZ, nU, nV;
    int pitch;            // row pitch of proj in elements
    int BU, BV;           // patch box
    float dVZ;
    float scale;
    int accumulate;       // add into the existing volume instead of overwriting it
    int skip_view;        // failure-detection test: no copy is issued for this local view (-1: none)
    int nsplit;           // blocks (one cluster) that share a tile's views
};

__device__ __forceinline__ uint32_t smem_u32(const void* p) {
    return (uint32_t)__cvta_generic_to_shared(p);
}

__device__ __forceinline__ bool mbar_wait(uint32_t bar, uint32_t phase) {
    for (unsigned i = 0; i < kWaitLimit; ++i) {
        uint32_t ok;
        asm volatile(
            "{\n\t.reg .pred p;\n\t"
            "mbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
            "selp.u32 %0, 1, 0, p;\n\t}"
            : "=r"(ok)
            : "r"(bar), "r"(phase)
            : "memory");
        if (ok) return true;
        __nanosleep(32);
    }
    return false;
}

// A tap of the patch.  The compiler may order it freely among the arithmetic; that it stays between the wait for
// the view's copy and the barrier behind which the patch is rewritten is seen to there: its address comes from
// a value made after the wait, and the sums are asked for before the barrier (volatile loads that
// clobber memory instead: 0.7 % on 181 x 203 x 190 tilted).
__device__ __forceinline__ float lds(uint32_t a) {
    float v;
    asm("ld.shared.f32 %0, [%1];" : "=f"(v) : "r"(a));
    return v;
}

__device__ __forceinline__ float2 f2(float a, float b) { return make_float2(a, b); }
__device__ __forceinline__ float2 f2(float a) { return make_float2(a, a); }
__device__ __forceinline__ float2 neg2(float2 a) { return make_float2(-a.x, -a.y); }
// a + t (b - a), two lanes at once
__device__ __forceinline__ float2 lerp2(float2 a, float2 b, float2 t) {
    return __ffma2_rn(t, __ffma2_rn(a, f2(-1.f), b), a);
}

// 1 / a by the hardware's approximation (relative error below 2^-22)
__device__ __forceinline__ float rcp_approx(float a) {
    float r;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(a));
    return r;
}

// texel-space (u - 0.5, v - 0.5) projection of voxel (x, y, z) for view frame F
__device__ __forceinline__ void project_texel(const FrameBPK& F, float x, float y, float z, float& ub, float& vb) {
    const double vx = fma((double)z, F.dz[0], fma((double)y, F.dy[0], fma((double)x, F.dx[0], F.b[0])));
    const double vy = fma((double)z, F.dz[1], fma((double)y, F.dy[1], fma((double)x, F.dx[1], F.b[1])));
    const double vz = fma((double)z, F.dz[2], fma((double)y, F.dy[2], fma((double)x, F.dx[2], F.b[2])));
    const float t = F.tnum / (float)vx;
    ub = fmaf((float)vy, t, F.cu) - 0.5f;
    vb = fmaf((float)vz, t, F.cv) - 0.5f;
}

// Warp 0: bounding box of the block's 8 corner voxels for local view la; lane 0 writes
// info[] and issues the TMA load (or a plain arrive when the box does not fit), unless
// `stopped` (lane 0's own wait for an earlier view expired: the buffer may still be awaiting
// that copy, so its barrier must not be re-armed).
__device__ __forceinline__ void plan_patch(const BPKArgs& p, const CUtensorMap* tmap, int la, int x0, int y0, int z0,
                                           float* dst, uint32_t bar, int* info, bool stopped) {
    const int lane = threadIdx.x & 31;
    const FrameBPK& F = p.frames[p.a0 + la];
    float ub = 0.f, vb = 0.f;
    if (lane < 8) {
        const int x = min(x0 + ((lane & 1) ? TXY - 1 : 0), p.nX - 1);
        const int y = min(y0 + ((lane & 2) ? TXY - 1 : 0), p.nY - 1);
        const int z = min(z0 + ((lane & 4) ? VZ - 1 : 0), p.nZ - 1);
        project_texel(F, (float)x, (float)y, (float)z, ub, vb);
    }
    float umin = lane < 8 ? ub : 3e38f, umax = lane < 8 ? ub : -3e38f;
    float vmin = lane < 8 ? vb : 3e38f, vmax = lane < 8 ? vb : -3e38f;
#pragma unroll
    for (int o = 4; o > 0; o >>= 1) {
        umin = fminf(umin, __shfl_xor_sync(0xffffffffu, umin, o));
        umax = fmaxf(umax, __shfl_xor_sync(0xffffffffu, umax, o));
        vmin = fminf(vmin, __shfl_xor_sync(0xffffffffu, vmin, o));
        vmax = fmaxf(vmax, __shfl_xor_sync(0xffffffffu, vmax, o));
    }
    if (lane == 0) {
        if (stopped) return;
        constexpr int ALIGN = 4;   // TMA: x * sizeof(float) a multiple of 16 bytes
        bool fits = isfinite(umin) && isfinite(umax) && isfinite(vmin) && isfinite(vmax) &&
                    fabsf(umin) < 1e7f && fabsf(vmin) < 1e7f;
        int u0 = 0, v0 = 0;
        if (fits) {
            u0 = (int)floorf(umin) - 1;
            u0 = (u0 >= 0) ? (u0 / ALIGN) * ALIGN : -(((-u0) + ALIGN - 1) / ALIGN) * ALIGN;
            v0 = (int)floorf(vmin) - 1;
            fits = ((int)ceilf(umax) + 2 - u0 <= p.BU - 1) && ((int)ceilf(vmax) + 2 - v0 <= p.BV - 1);
        }
        info[0] = u0;
        info[1] = v0;
        info[2] = fits ? 1 : 0;
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        if (la == p.skip_view) {
            // failure-detection test: neither a copy nor an arrival, so the wait for this view
            // runs out with nothing in flight
        } else if (fits) {
            const uint32_t bytes = (uint32_t)(p.BU * p.BV * sizeof(float));
            asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
            asm volatile(
                "cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], "
                "[%5];" ::"r"(smem_u32(dst)),
                "l"((unsigned long long)tmap), "r"(u0), "r"(v0), "r"(la), "r"(bar)
                : "memory");
        } else {
            asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
        }
    }
}

__device__ __forceinline__ float global_sample(const BPKArgs& p, const float* P, float ub, float vb) {
    const float fx = floorf(ub), fy = floorf(vb);
    const float au = ub - fx, av = vb - fy;
    const int iu = (int)fmaxf(fminf(fx, 1e8f), -1e8f), iv = (int)fmaxf(fminf(fy, 1e8f), -1e8f);
    auto at = [&](int u, int v) -> float {
        return (u >= 0 && u < p.nU && v >= 0 && v < p.nV) ? P[(long)v * p.pitch + u] : 0.f;
    };
    const float a0 = fmaf(au, at(iu + 1, iv) - at(iu, iv), at(iu, iv));
    const float a1 = fmaf(au, at(iu + 1, iv + 1) - at(iu, iv + 1), at(iu, iv + 1));
    return fmaf(av, a1 - a0, a0);
}

template <typename TV, bool MATCHED, bool AXIAL, bool SPLIT>
__global__ void __launch_bounds__(TXY* TXY, 2) bp_tma_kernel(const __grid_constant__ CUtensorMap tmap, BPKArgs p) {
    extern __shared__ __align__(128) unsigned char smem_raw[];
    __shared__ __align__(8) unsigned long long bars[2];
    __shared__ int info[2][4];
    __shared__ int tile_failed;   // SPLIT: a wait of this block expired
    // SPLIT: the blocks of a cluster (along z) own one tile and views [lb, lb + nviews) of it each
    const int rank = SPLIT ? (int)(blockIdx.z % (unsigned)p.nsplit) : 0;
    const int lb = SPLIT ? (int)((long)p.na * rank / p.nsplit) : 0;
    const int nviews = (SPLIT ? (int)((long)p.na * (rank + 1) / p.nsplit) : p.na) - lb;
    // TMA destinations: 128-byte aligned, each buffer rounded up to 128 bytes
    const uint32_t base_off = (128u - (smem_u32(smem_raw) & 127u)) & 127u;
    const size_t buf_bytes = ((size_t)p.BU * p.BV * sizeof(float) + 127) / 128 * 128;
    float* buf0 = reinterpret_cast<float*>(smem_raw + base_off);
    float* buf1 = reinterpret_cast<float*>(smem_raw + base_off + buf_bytes);
    const uint32_t buf0_u32 = smem_u32(buf0), buf1_u32 = smem_u32(buf1);
    const uint32_t rowb = (uint32_t)(p.BU * sizeof(float));
    const int tid = threadIdx.x;
    // each warp covers an 8 x 4 patch of columns: at every view angle its 32 samples of one
    // slice fall on a compact set of detector texels (few shared-memory wavefronts)
    const int wid = tid >> 5, ln = tid & 31;
    const int tx = (wid & 1) * 8 + (ln & 7), ty = (wid >> 1) * 4 + (ln >> 3);
    const int x0 = blockIdx.x * TXY, y0 = blockIdx.y * TXY;
    const int z0 = (int)(SPLIT ? blockIdx.z / (unsigned)p.nsplit : blockIdx.z) * VZ;
    const int x = x0 + tx, y = y0 + ty;
    const bool active = x < p.nX && y < p.nY;
    const uint32_t bar0 = smem_u32(&bars[0]), bar1 = smem_u32(&bars[1]);
    if (tid == 0) {
        asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(bar0) : "memory");
        asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(bar1) : "memory");
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        tile_failed = 0;
    }
    __syncthreads();
    if (tid < 32) {
        plan_patch(p, &tmap, lb, x0, y0, z0, buf0, bar0, info[0], false);
        if (nviews > 1) plan_patch(p, &tmap, lb + 1, x0, y0, z0, buf1, bar1, info[1], false);
    }
    float acc[VZ];
#pragma unroll
    for (int k = 0; k < VZ; ++k) acc[k] = 0.f;
    const float* Pg = (const float*)p.proj;
    const float pumax = (float)(p.BU - 2), pvmax = (float)(p.BV - 2);
    int failed_at = -1;   // first view (of this block's) whose wait expired in this thread
    for (int i = 0; i < nviews; ++i) {
        const int la = lb + i;
        const int s = i & 1;
        const uint32_t bar = s ? bar1 : bar0;
        // after one expired wait this thread waits no more (its sums are not written)
        if (failed_at < 0 && !mbar_wait(bar, (uint32_t)((i >> 1) & 1))) failed_at = i;
        const float* patch = s ? buf1 : buf0;
        uint32_t patch_u32 = s ? buf1_u32 : buf0_u32;
        asm volatile("" : "+r"(patch_u32) : : "memory");           // lds: no tap before here
        const int u0 = info[s][0], v0 = info[s][1], fits = info[s][2];
        if (active) {
            const FrameBPK& F = p.frames[p.a0 + la];
            const double bxd = fma((double)z0, F.dz[0], fma((double)y, F.dy[0], fma((double)x, F.dx[0], F.b[0])));
            const double byd = fma((double)z0, F.dz[1], fma((double)y, F.dy[1], fma((double)x, F.dx[1], F.b[1])));
            const double bzd = fma((double)z0, F.dz[2], fma((double)y, F.dy[2], fma((double)x, F.dx[2], F.b[2])));
            const float vx = (float)bxd, vy = (float)byd, vz = (float)bzd;
            float wcol = 1.f, cu2 = 0.f, cxy = 0.f;
            if (!MATCHED) {
                const float den = fmaf((float)y, F.wy, fmaf((float)x, F.wx, F.w0));
                const float r = __fdividef(F.dso, den);
                wcol = r * r;
            } else {
                const float rvx = fmaf((float)x, F.dvx, F.rv0x), rvy = fmaf((float)y, F.dvy, F.rv0y);
                cxy = (F.rsx - rvx) * (F.rsx - rvx) + (F.rsy - rvy) * (F.rsy - rvy);
            }
            if (AXIAL) {
                const float t = F.tnum / vx;
                const float u = fmaf(vy, t, F.cu);            // texture coordinate
                const float vt0 = fmaf(vz, t, F.cv);
                const float vstep = (float)F.dz[2] * t;
                if (MATCHED) {
                    const float day = fmaf(u, F.ddu, F.du0);
                    const float dx = fmaf(day, F.sina, F.daxc), dy = fmaf(day, F.cosa, -F.daxs);
                    cu2 = (F.rsx - dx) * (F.rsx - dx) + (F.rsy - dy) * (F.rsy - dy);
                }
                if (fits) {
                    const float pu = fminf(fmaxf(u - 0.5f - (float)u0, 0.f), pumax);
                    const int iu = (int)pu;
                    const float2 fu2 = f2(pu - (float)iu);
                    const float pv0 = vt0 - 0.5f - (float)v0;
                    constexpr uint32_t ES = (uint32_t)sizeof(float);
                    const uint32_t colb = patch_u32 + (uint32_t)iu * ES;
                    const float2 vstep2 = f2(vstep);
                    const float2 pv02 = f2(pv0);
                    const float2 w2 = f2(wcol);
                    // rows stay inside the patch for the whole column -> no per-voxel clamps
                    const float pvlast = fmaf((float)(VZ - 1), vstep, pv0);
                    const bool inside = fminf(pv0, pvlast) >= 0.f && fmaxf(pv0, pvlast) <= pvmax;
                    // Matched weight w(k) = L^3 / (DSD lsq) along the column: L^2 and lsq are
                    // quadratics in the slice index k with complex roots hundreds of slices away,
                    // so w is interpolated by the cubic through its exact values at the four
                    // Chebyshev nodes of [0, VZ-1] (relative error ~1e-7 at a 6:10 source/detector
                    // distance ratio, far below that at the usual ones).  In s = k - (VZ-1)/2,
                    // with nodes +-na, +-nb, the cubic is e0 + o1 s + e2 s^2 + o3 s^3.  The node
                    // values use the hardware reciprocal square root and the approximate
                    // division (each within 2 ulp), since they run once per column and view.
                    float2 c0 = f2(0.f), c1 = f2(0.f), c2 = f2(0.f), c3 = f2(0.f);
                    if (MATCHED) {
                        constexpr float hw = 0.5f * (float)(VZ - 1);
                        constexpr float na = hw * 0.92387953251f;   // cos(pi/8) = sqrt(2 + sqrt 2) / 2
                        constexpr float nb = hw * 0.38268343236f;   // cos(3pi/8) = sqrt(2 - sqrt 2) / 2
                        constexpr float inv = 1.f / (na * na - nb * nb);
                        const float rz0 = fmaf((float)z0, p.dVZ, F.rv0z);
                        auto wexact = [&](float kf) {
                            const float vt = fmaf(kf, vstep, vt0), dz = fmaf(vt, F.ddv, F.dzc), L2 = fmaf(dz, dz, cu2);
                            const float rvz = fmaf(kf, p.dVZ, rz0), lsq = fmaf(rvz, rvz, cxy);
                            return __fdividef(L2 * L2 * rsqrtf(L2), F.dsd * lsq);
                        };
                        const float wpa = wexact(hw + na), wma = wexact(hw - na);
                        const float wpb = wexact(hw + nb), wmb = wexact(hw - nb);
                        const float Ea = 0.5f * (wpa + wma), Eb = 0.5f * (wpb + wmb);
                        const float Oa = (wpa - wma) * (0.5f / na), Ob = (wpb - wmb) * (0.5f / nb);
                        const float e2 = (Ea - Eb) * inv, o3 = (Oa - Ob) * inv;
                        c0 = f2(fmaf(-e2, na * na, Ea));
                        c1 = f2(fmaf(-o3, na * na, Oa));
                        c2 = f2(e2);
                        c3 = f2(o3);
                    }
                    // the float bits of the floor below index the patch directly:
                    // row address = bits * rowb + colb - 0x4B400000 * rowb (32-bit wrap)
                    const uint32_t colb_m = colb - 0x4B400000u * rowb;
                    auto pairs = [&](auto clamp_tag) {
                        constexpr bool CLAMP = decltype(clamp_tag)::value;
#pragma unroll
                        for (int k = 0; k < VZ; k += 2) {
                            const float2 kk = f2((float)k, (float)(k + 1));
                            float2 pv = __ffma2_rn(kk, vstep2, pv02);
                            if (CLAMP) {
                                pv.x = fminf(fmaxf(pv.x, 0.f), pvmax);
                                pv.y = fminf(fmaxf(pv.y, 0.f), pvmax);
                            }
                            // floor / fraction with packed arithmetic: pv >= 0 here, and at 1.5*2^23
                            // the float spacing is 1, so a round-toward-zero add of 1.5*2^23 leaves
                            // floor(pv) in the low mantissa bits; subtracting it back is exact
                            const float2 t = __fadd2_rz(pv, f2(12582912.0f));
                            const float2 fv = __ffma2_rn(__fadd2_rn(t, f2(-12582912.0f)), f2(-1.f), pv);
                            const uint32_t aa = (uint32_t)__float_as_int(t.x) * rowb + colb_m;
                            const uint32_t ab = (uint32_t)__float_as_int(t.y) * rowb + colb_m;
                            const float2 r0 = f2(lds(aa), lds(ab)), r0r = f2(lds(aa + ES), lds(ab + ES));
                            const float2 r1 = f2(lds(aa + rowb), lds(ab + rowb));
                            const float2 r1r = f2(lds(aa + rowb + ES), lds(ab + rowb + ES));
                            const float2 smp = lerp2(lerp2(r0, r0r, fu2), lerp2(r1, r1r, fu2), fv);
                            float2 w = w2;
                            if (MATCHED) {
                                const float2 s2 = f2((float)k - 0.5f * (float)(VZ - 1), (float)(k + 1) - 0.5f * (float)(VZ - 1));
                                w = __ffma2_rn(__ffma2_rn(__ffma2_rn(c3, s2, c2), s2, c1), s2, c0);
                            }
                            const float2 acc2 = __ffma2_rn(smp, w, f2(acc[k], acc[k + 1]));
                            acc[k] = acc2.x;
                            acc[k + 1] = acc2.y;
                        }
                    };
                    if (inside) pairs(std::false_type{});
                    else pairs(std::true_type{});
                } else {
                    // unrolled: a runtime index into acc[] would move it to local memory
#pragma unroll
                    for (int k = 0; k < VZ; ++k) {
                        const float vtex = fmaf((float)k, vstep, vt0);
                        const float smp = global_sample(p, Pg + (long)la * p.pitch * p.nV, u - 0.5f, vtex - 0.5f);
                        float w = wcol;
                        if (MATCHED) {
                            const float dz = fmaf(vtex, F.ddv, F.dzc);
                            const float L2 = fmaf(dz, dz, cu2);
                            const float rvz = fmaf((float)(z0 + k), p.dVZ, F.rv0z);
                            const float lsq = fmaf(rvz, rvz, cxy);
                            w = L2 * (L2 * rsqrtf(L2)) * __frcp_rn(F.dsd * lsq);
                        }
                        acc[k] = fmaf(smp, w, acc[k]);
                    }
                }
            } else {
                // Tilted frames: u, v and the depth all change along a column, so each voxel has
                // its own reciprocal (hardware approximation and one Newton step) and horizontal
                // fraction; otherwise the packed arithmetic of the axial path, two slices at
                // a time.  The projective map keeps the order along a column, so when both of its
                // ends fall inside the patch all of it does and no coordinate is clamped.
                // 181 x 203 x 190 voxels, 77 views of 233 x 251, matched, one block a tile: 4218 -> 1170 us (an IEEE division,
                // clamps, an unpacked sample and 90 instructions per voxel before); bound by issue.
                const float dzx = (float)F.dz[0], dzy = (float)F.dz[1], dzz = (float)F.dz[2];
                if (fits) {
                    const float cup = F.cu - 0.5f - (float)u0, cvp = F.cv - 0.5f - (float)v0;   // patch coordinates
                    constexpr uint32_t ES = (uint32_t)sizeof(float);
                    const uint32_t base = patch_u32 - 0x4B400000u * rowb - 0x4B400000u * ES;
                    const float cw = 0.5f + (float)u0, cz = 0.5f + (float)v0;
                    const float day0 = fmaf(cw, F.ddu, F.du0), dz0 = fmaf(cz, F.ddv, F.dzc);
                    const float dx0 = F.daxc - F.rsx, dy0 = -F.daxs - F.rsy;
                    const float rz0 = fmaf((float)z0, p.dVZ, F.rv0z);
                    bool inside = true;
#pragma unroll
                    for (int e = 0; e < 2; ++e) {
                        const float kf = e ? (float)(VZ - 1) : 0.f;
                        const float ex = fmaf(kf, dzx, vx), t = __fdividef(F.tnum, ex);
                        const float ue = fmaf(fmaf(kf, dzy, vy), t, cup), ve = fmaf(fmaf(kf, dzz, vz), t, cvp);
                        inside = inside && t > 0.f && ue >= 0.25f && ue <= pumax - 0.25f && ve >= 0.25f && ve <= pvmax - 0.25f;
                    }
                    auto pairs = [&](auto clamp_tag) {
                        constexpr bool CLAMP = decltype(clamp_tag)::value;
#pragma unroll
                        for (int k = 0; k < VZ; k += 2) {
                            const float2 kk = f2((float)k, (float)(k + 1));
                            const float2 ex = __ffma2_rn(kk, f2(dzx), f2(vx));
                            float2 r = f2(rcp_approx(ex.x), rcp_approx(ex.y));
                            r = __ffma2_rn(__ffma2_rn(neg2(ex), r, f2(1.f)), r, r);
                            const float2 t = __fmul2_rn(f2(F.tnum), r);
                            float2 pu = __ffma2_rn(__ffma2_rn(kk, f2(dzy), f2(vy)), t, f2(cup));
                            float2 pv = __ffma2_rn(__ffma2_rn(kk, f2(dzz), f2(vz)), t, f2(cvp));
                            if (CLAMP) {
                                pu.x = fminf(fmaxf(pu.x, 0.f), pumax);
                                pu.y = fminf(fmaxf(pu.y, 0.f), pumax);
                                pv.x = fminf(fmaxf(pv.x, 0.f), pvmax);
                                pv.y = fminf(fmaxf(pv.y, 0.f), pvmax);
                            }
                            // floors and fractions as on the axial path, for both coordinates
                            const float2 tu = __fadd2_rz(pu, f2(12582912.0f)), tv = __fadd2_rz(pv, f2(12582912.0f));
                            const float2 fu = __ffma2_rn(__fadd2_rn(tu, f2(-12582912.0f)), f2(-1.f), pu);
                            const float2 fv = __ffma2_rn(__fadd2_rn(tv, f2(-12582912.0f)), f2(-1.f), pv);
                            const uint32_t aa = (uint32_t)__float_as_int(tv.x) * rowb + ((uint32_t)__float_as_int(tu.x) * ES + base);
                            const uint32_t ab = (uint32_t)__float_as_int(tv.y) * rowb + ((uint32_t)__float_as_int(tu.y) * ES + base);
                            const float2 r0 = f2(lds(aa), lds(ab)), r0r = f2(lds(aa + ES), lds(ab + ES));
                            const float2 r1 = f2(lds(aa + rowb), lds(ab + rowb));
                            const float2 r1r = f2(lds(aa + rowb + ES), lds(ab + rowb + ES));
                            const float2 smp = lerp2(lerp2(r0, r0r, fu), lerp2(r1, r1r, fu), fv);
                            float2 w = f2(wcol);
                            if (MATCHED) {
                                const float2 day = __ffma2_rn(pu, f2(F.ddu), f2(day0)), dz = __ffma2_rn(pv, f2(F.ddv), f2(dz0));
                                const float2 dx = __ffma2_rn(day, f2(F.sina), f2(dx0)), dy = __ffma2_rn(day, f2(F.cosa), f2(dy0));
                                const float2 L2 = __ffma2_rn(dz, dz, __ffma2_rn(dy, dy, __fmul2_rn(dx, dx)));
                                const float2 rvz = __ffma2_rn(kk, f2(p.dVZ), f2(rz0));
                                const float2 q = __fmul2_rn(f2(F.dsd), __ffma2_rn(rvz, rvz, f2(cxy)));
                                const float2 L3 = __fmul2_rn(__fmul2_rn(L2, f2(rsqrtf(L2.x), rsqrtf(L2.y))), L2);
                                w = __fmul2_rn(L3, f2(rcp_approx(q.x), rcp_approx(q.y)));
                            }
                            const float2 acc2 = __ffma2_rn(smp, w, f2(acc[k], acc[k + 1]));
                            acc[k] = acc2.x;
                            acc[k + 1] = acc2.y;
                        }
                    };
                    if (inside) pairs(std::false_type{});
                    else pairs(std::true_type{});
                } else {
#pragma unroll
                    for (int k = 0; k < VZ; ++k) {
                        const float kf = (float)k;
                        const float ex = fmaf(kf, dzx, vx), ey = fmaf(kf, dzy, vy), ez = fmaf(kf, dzz, vz);
                        const float t = F.tnum / ex;
                        const float u = fmaf(ey, t, F.cu), vtex = fmaf(ez, t, F.cv);
                        const float smp = global_sample(p, Pg + (long)la * p.pitch * p.nV, u - 0.5f, vtex - 0.5f);
                        float w = wcol;
                        if (MATCHED) {
                            const float day = fmaf(u, F.ddu, F.du0);
                            const float dx = fmaf(day, F.sina, F.daxc), dy = fmaf(day, F.cosa, -F.daxs);
                            const float dz = fmaf(vtex, F.ddv, F.dzc);
                            const float L2 = (F.rsx - dx) * (F.rsx - dx) + (F.rsy - dy) * (F.rsy - dy) + dz * dz;
                            const float rvz = fmaf((float)(z0 + k), p.dVZ, F.rv0z);
                            const float lsq = fmaf(rvz, rvz, cxy);
                            w = L2 * (L2 * rsqrtf(L2)) * __frcp_rn(F.dsd * lsq);
                        }
                        acc[k] = fmaf(smp, w, acc[k]);
                    }
                }
            }
        }
#pragma unroll
        for (int k = 0; k < VZ; ++k) asm volatile("" : : "f"(acc[k]) : "memory");   // lds: no tap behind here
        __syncthreads();   // everyone is done with buffer s
        if (tid < 32 && i + 2 < nviews) plan_patch(p, &tmap, la + 2, x0, y0, z0, s ? buf1 : buf0, bar, info[s], failed_at >= 0);
    }
    if (tid == 0 && failed_at >= 0) {
        // thread 0 issued nothing after its failed view: the copies of that view and the next
        // may still be in flight, so wait for them (bounded) before the block's shared memory
        // is released
        for (int v = failed_at; v < min(failed_at + 2, nviews); ++v)
            if (lb + v != p.skip_view) mbar_wait((v & 1) ? bar1 : bar0, (uint32_t)((v >> 1) & 1));
    }
    if constexpr (SPLIT) {
        namespace cg = cooperative_groups;
        cg::cluster_group cluster = cg::this_cluster();
        // this block's sums replace its patches (every warp is past the last view's barrier);
        // a failed block still reaches both cluster barriers, and its tile is not written
        float* sums = reinterpret_cast<float*>(smem_raw + base_off);   // [VZ][TXY * TXY]
#pragma unroll
        for (int k = 0; k < VZ; ++k) sums[k * TXY * TXY + tid] = acc[k];
        if (failed_at >= 0) {
            tile_failed = 1;
            if (p.status) atomicOr(p.status, TIGRE_STATUS_WAIT_EXPIRED);
        }
        cluster.sync();
        int bad = 0;
#pragma unroll
        for (int r = 0; r < kMaxSplit; ++r)
            if (r < p.nsplit) bad |= *cluster.map_shared_rank(&tile_failed, r);
        if (active && !bad) {
            TV* V = (TV*)p.vol;
            const int kend = min(VZ * (rank + 1) / p.nsplit, p.nZ - z0);
#pragma unroll 2
            for (int k = VZ * rank / p.nsplit; k < kend; ++k) {
                // every block's value is requested before the first is used
                float v[kMaxSplit];
#pragma unroll
                for (int r = 0; r < kMaxSplit; ++r)
                    v[r] = r < p.nsplit ? cluster.map_shared_rank(sums, r)[k * TXY * TXY + tid] : 0.f;
                float t = v[0];
#pragma unroll
                for (int r = 1; r < kMaxSplit; ++r) t += v[r];
                const size_t i = ((size_t)(z0 + k) * p.nY + y) * p.nX + x;
                const float o = p.accumulate ? to_f32<TV>(V[i]) : 0.f;
                V[i] = from_f32<TV>(fmaf(t, p.scale, o));
            }
        }
        cluster.sync();   // the sums stay until every block of the cluster has read them
        return;
    }
    if (__any_sync(0xffffffffu, failed_at >= 0)) {
        if ((tid & 31) == 0 && p.status) atomicOr(p.status, TIGRE_STATUS_WAIT_EXPIRED);
        return;
    }
    if (!active) return;
    TV* V = (TV*)p.vol;
#pragma unroll
    for (int k = 0; k < VZ; ++k) {
        const int z = z0 + k;
        if (z < p.nZ) {
            const size_t i = ((size_t)z * p.nY + y) * p.nX + x;
            const float o = p.accumulate ? to_f32<TV>(V[i]) : 0.f;
            V[i] = from_f32<TV>(fmaf(acc[k], p.scale, o));
        }
    }
}

PFN_cuTensorMapEncodeTiled_v12000 encode_fn() {
    static PFN_cuTensorMapEncodeTiled_v12000 fn = nullptr;
    static std::once_flag once;
    std::call_once(once, [] {
        void* f = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &f, cudaEnableDefault, &q) == cudaSuccess &&
            q == cudaDriverEntryPointSuccess)
            fn = reinterpret_cast<PFN_cuTensorMapEncodeTiled_v12000>(f);
    });
    return fn;
}

// Blocks per tile, a power of two up to 8 (the portable cluster size), from the time that the
// rounds of resident blocks take, as measured over 15 volumes of 16^3 to 200^3, 4 to 180 views and each
// number of blocks: a view costs a block 2.4 us alone on an SM and 3.9 when two share it (matched; FDK 2.5 and
// 3.45), the call 6 us beside the views, 13 with the exchange of the sums, and a further round 6.  Sharing is
// taken from four views a block on and where it saves 5 % in this account (9 % for the eighth
// block, whose clusters pack worse).  Over the 330 entries no choice is more than 1 % slower than one
// block a tile.  Matched, one block -> chosen: 64^3 with 100 views 247 -> 63 us (8 blocks), with 16 46 -> 20 (4),
// 96^3 / 60 153 -> 106 (4), 128^3 / 180 441 -> 381 (2) and / 12 38 (1; two blocks 40), 160^3 / 100 608 -> 471 (4).
int bp_splits(long blocks, int na, bool matched) {
    constexpr long kSms = 148, kSlots = 2 * kSms;
    const double alone = matched ? 2.4 : 2.5, shared = matched ? 3.9 : 3.45;
    int best = 1;
    double best_t = 0.0;
    for (int s = 1; s <= kMaxSplit; s *= 2) {
        if (s > 1 && na < 4 * s) break;
        const int views = (na + s - 1) / s;
        const long full = blocks * s / kSlots, rest = blocks * s % kSlots;
        double t = (s == 1 ? 6.0 : 13.0) + 6.0 * (double)(full + (rest > 0) - 1) + (double)full * shared * views;
        if (rest) t += (rest > kSms ? shared : alone) * views;
        if (s == 1 || t < (s == 8 ? 0.91 : 0.95) * best_t) { best = s; best_t = t; }
    }
    return best;
}

template <typename TV>
int launch_typed(const CUtensorMap& tm, BPKArgs a, bool matched, bool axial, cudaStream_t st) {
    dim3 grid((a.nX + TXY - 1) / TXY, (a.nY + TXY - 1) / TXY, (a.nZ + VZ - 1) / VZ);
    a.nsplit = bp_splits((long)grid.x * grid.y * grid.z, a.na, matched);
    size_t smem = 2 * (((size_t)a.BU * a.BV * sizeof(float) + 127) / 128 * 128) + 128;
    auto go = [&](auto kern) -> int {
        TIGRE_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
        kern<<<grid, TXY * TXY, smem, st>>>(tm, a);
        TIGRE_LAUNCHED();
        return TIGRE_SUCCESS;
    };
    auto go_split = [&](auto kern) -> int {
        smem = std::max(smem, (size_t)VZ * TXY * TXY * sizeof(float) + 128);
        TIGRE_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
        cudaLaunchAttribute attr{};
        attr.id = cudaLaunchAttributeClusterDimension;
        attr.val.clusterDim.x = attr.val.clusterDim.y = 1;
        attr.val.clusterDim.z = (unsigned)a.nsplit;
        cudaLaunchConfig_t cfg{};
        cfg.gridDim = dim3(grid.x, grid.y, grid.z * (unsigned)a.nsplit);
        cfg.blockDim = dim3(TXY * TXY);
        cfg.dynamicSmemBytes = smem;
        cfg.stream = st;
        cfg.attrs = &attr;
        cfg.numAttrs = 1;
        TIGRE_CUDA(cudaLaunchKernelEx(&cfg, kern, tm, a));
        TIGRE_LAUNCHED();
        return TIGRE_SUCCESS;
    };
    if (a.nsplit > 1) {
        if (matched) return axial ? go_split(bp_tma_kernel<TV, true, true, true>) : go_split(bp_tma_kernel<TV, true, false, true>);
        return axial ? go_split(bp_tma_kernel<TV, false, true, true>) : go_split(bp_tma_kernel<TV, false, false, true>);
    }
    if (matched) return axial ? go(bp_tma_kernel<TV, true, true, false>) : go(bp_tma_kernel<TV, true, false, false>);
    return axial ? go(bp_tma_kernel<TV, false, true, false>) : go(bp_tma_kernel<TV, false, false, false>);
}

}  // namespace

bool bp_tma_supported(const TigrePlan* P) {
    return P->bp_box_u > 0 && encode_fn() != nullptr;
}

int launch_backproject_tma(TigrePlan* P, const float* proj, int pitch, void* vol, int vdt, int matched, int a0, int a1,
                           int accumulate, cudaStream_t st) {
    auto enc = encode_fn();
    if (!enc) return fail(TIGRE_ERR_CUDA, "cuTensorMapEncodeTiled unavailable");
    const int na = a1 - a0;
    const size_t es = sizeof(float);
    CUtensorMap tm;
    cuuint64_t dims[3] = {(cuuint64_t)pitch, (cuuint64_t)P->d.nV, (cuuint64_t)na};
    cuuint64_t strides[2] = {(cuuint64_t)pitch * es, (cuuint64_t)pitch * P->d.nV * es};
    const int BU = P->bp_box_u;
    cuuint32_t box[3] = {(cuuint32_t)BU, (cuuint32_t)P->bp_box_v, 1};
    cuuint32_t estr[3] = {1, 1, 1};
    CUresult r = enc(&tm, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 3,
                     const_cast<float*>(proj), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                     CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) return fail(TIGRE_ERR_CUDA, "cuTensorMapEncodeTiled failed");
    BPKArgs a{};
    a.frames = P->d_bpk;
    a.proj = proj;
    a.vol = vol;
    a.status = P->d_status;
    a.a0 = a0;
    a.na = na;
    a.nX = P->d.nX; a.nY = P->d.nY; a.nZ = P->d.nZ; a.nU = P->d.nU; a.nV = P->d.nV;
    a.pitch = pitch;
    a.BU = BU;
    a.BV = P->bp_box_v;
    a.dVZ = (float)P->d.dVZ;
    a.scale = matched ? (float)(P->d.dVX * P->d.dVY * P->d.dVZ / (P->d.dDU * P->d.dDV)) : 1.f;
    a.accumulate = accumulate;
    const long long skip = option(TIGRE_OPT_BP_SKIP_COPY);
    a.skip_view = (skip >= 0 && skip < na) ? (int)skip : -1;
    const bool ax = P->axial;
    if (vdt == TIGRE_F32) return launch_typed<float>(tm, a, matched, ax, st);
    return launch_typed<__nv_bfloat16>(tm, a, matched, ax, st);
}

}  // namespace tigre
