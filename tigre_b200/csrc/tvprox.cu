// TV proximal operator (ROF denoising by a primal-dual iteration), sm_100a.
//
// Same iteration as tvdenoising (Common/CUDA/tv_proximal.cu:185-630) on one device:
//   u = f, p = 0; for i < maxIter:
//     tau2 = 0.3 + 0.02 i,  tau1 = (1/tau2) (1/6 - 5/(15 + i))
//     u <- (1 - tau1) u + tau1 (f + div(p) / lambda)          (update_u, :136-153)
//     q = p + tau2 grad(u);  p <- q / max(1, |q|)              (update_p, :156-181)
// with backward-difference divergence (p taken as 0 before index 0, :81-109) and
// forward-difference gradient (0 at the last index, :111-134), each divided by the spacing.
// The volume is iterated with one extra slice below and above in z, as the reference's
// single-device layout does (buffer_length = 1): the lower one holds slice 1 of the image,
// the upper one zeros (cpy_from_host, :672-692, writes its mirror slice where the image
// copy then lands), and both evolve with the rest.
//
// Two forms.  With 8 (nZ + 2) nY nX floats of work space (tigre_tv_denoise_ex) an iteration is
// one pass, prox_step_kernel: u and p are kept twice, and a warp marching down the slices
// recomputes the u of the +x, +y and +z neighbours that its p needs.  It reads f, u and p and
// writes u and p once, 36 bytes per voxel; the image itself stands for f, the first pass needs no
// initialised state and the last one writes only the result.
// With 5 (nZ + 2) nY nX floats, for volumes whose doubled state does not fit, f, u, px, py and pz
// are (nZ + 2, nY, nX) arrays in the work buffer and an iteration is two passes
// (prox_update_u, prox_update_p), 52 bytes per voxel.

#include <climits>
#include <cmath>

#include "tigre_internal.h"

namespace tigre {
namespace {

struct ProxDims {
    int nx, ny, nzp;         // nzp = nZ + 2
    float idx, idy, idz;     // 1 / spacing
};

// Voxels of the (nzp, ny, nx) arrays: blocks stride over (y, z) rows, threads over x, so no
// thread divides a linear index; i is the linear index of (x, y, z).
#define PROX_FOR_EACH_VOXEL(d, x, y, z, i)                                                   \
    for (long row_ = blockIdx.x; row_ < (long)(d).ny * (d).nzp; row_ += gridDim.x) {        \
        const int y = (int)(row_ % (d).ny), z = (int)(row_ / (d).ny);                         \
        for (int x = threadIdx.x; x < (d).nx; x += blockDim.x) {                               \
            const long i = row_ * (d).nx + x;
#define PROX_END_FOR_EACH_VOXEL \
    }                           \
    }

__global__ void __launch_bounds__(256) prox_update_u(const float* __restrict__ f, const float* __restrict__ pz,
                                                     const float* __restrict__ py, const float* __restrict__ px,
                                                     float* __restrict__ u, float tau, float inv_lambda, ProxDims d) {
    const long plane = (long)d.nx * d.ny;
    PROX_FOR_EACH_VOXEL(d, x, y, z, i) {
        float div = z > 0 ? (pz[i] - pz[i - plane]) * d.idz : pz[i];
        div += y > 0 ? (py[i] - py[i - d.nx]) * d.idy : py[i];
        div += x > 0 ? (px[i] - px[i - 1]) * d.idx : px[i];
        u[i] = u[i] * (1.f - tau) + tau * (f[i] + inv_lambda * div);
    }
    PROX_END_FOR_EACH_VOXEL
}

__global__ void __launch_bounds__(256) prox_update_p(const float* __restrict__ u, float* __restrict__ pz,
                                                     float* __restrict__ py, float* __restrict__ px, float tau,
                                                     ProxDims d) {
    const long plane = (long)d.nx * d.ny;
    PROX_FOR_EACH_VOXEL(d, x, y, z, i) {
        const float c = u[i];
        const float gz = z + 1 < d.nzp ? (u[i + plane] - c) * d.idz : 0.f;
        const float gy = y + 1 < d.ny ? (u[i + d.nx] - c) * d.idy : 0.f;
        const float gx = x + 1 < d.nx ? (u[i + 1] - c) * d.idx : 0.f;
        const float q0 = pz[i] + tau * gz, q1 = py[i] + tau * gy, q2 = px[i] + tau * gx;
        const float nrm = fmaxf(1.f, sqrtf(q0 * q0 + q1 * q1 + q2 * q2));
        pz[i] = q0 / nrm;
        py[i] = q1 / nrm;
        px[i] = q2 / nrm;
    }
    PROX_END_FOR_EACH_VOXEL
}

int grid_for_prox(const ProxDims& d) {
    return (int)std::min<long>((long)d.ny * d.nzp, 148L * 16);
}

// ---- one pass per iteration ----
//
// A warp owns 30 x kStepRows columns of a chunk of zc slices.  Lane l holds x = 30 bx + l - 1;
// lanes 0 and 31 only supply the neighbours' values (by shuffle), as row kStepRows does for +y,
// and u of slice z + 1 is formed one step ahead.  Per step and row that is five loads, no shared
// memory and no barrier; the rows re-read by the neighbouring warps of the block hit L1.
// Bound by the latency of its memory accesses (36 B per voxel; five loads a row in flight per
// warp).  One iteration: 256^3 120 us (the two passes 213), 512^3 934 us (1557), 301 x 333 x 317 222 us (514),
// 64^3 6 us (14).  4 rows at 5 blocks per SM; 4 / 6, 6 / 4 and 8 / 4: 985, 977 and 961 us at 512^3.
constexpr int kStepRows = 4, kStepWarps = 4, kStepLanes = 30, kStepBlocks = 5;

struct ProxStep {
    const float* src;               // the image (nZ slices); f is it between its halo slices
    const float *u, *pz, *py, *px;  // state in
    float *u_out, *pz_out, *py_out, *px_out;
    float tau1, tau2, inv_lambda;
    int zc;
};

// q / max(1, |q|) as a factor: 1 / |q| from the hardware reciprocal square root and one Newton
// step (error within 1.2 ulp, as a correctly rounded root and quotient together)
__device__ __forceinline__ float prox_shrink(float s) {
    if (!(s > 1.f)) return 1.f;
    if (!(s < 1e37f)) return 1.f / sqrtf(s);
    float r;
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(s));
    const float h = 0.5f * r, e = fmaf(-s * r, r, 1.f);
    return fmaf(h, e, r);
}

// FIRST: u = f and p = 0 are not read.  LAST: writes u only, as the (nZ, nY, nX) result.
// Off: type of the byte offsets within a slice (32 bits wherever a slice is below 4 GB).
template <bool FIRST, bool LAST, typename Off>
__global__ void __launch_bounds__(32 * kStepWarps, kStepBlocks) prox_step_kernel(ProxStep a, ProxDims d) {
    constexpr int R = kStepRows;
    const int tx = (d.nx + kStepLanes - 1) / kStepLanes, ty = (d.ny + R * kStepWarps - 1) / (R * kStepWarps);
    const int lane = threadIdx.x & 31, wid = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0);
    const int bx = (int)(blockIdx.x % (unsigned)tx), bt = (int)(blockIdx.x / (unsigned)tx);
    const int x = bx * kStepLanes + lane - 1, y0 = (bt % ty * kStepWarps + wid) * R;
    const int z0 = bt / ty * a.zc, zend = min(z0 + a.zc, d.nzp);
    if (y0 >= d.ny) return;
    const bool out = lane >= 1 && lane <= kStepLanes && x < d.nx;
    const float sx = x > 0 ? d.idx : 1.f, sy0 = y0 > 0 ? d.idy : 1.f;
    const float ix = x + 1 < d.nx ? d.idx : 0.f;
    const size_t plane = (size_t)d.nx * d.ny;
    // byte offsets in a slice of rows y0-1 .. y0+R, clamped to the volume (clamped values are not used)
    const Off xc = (Off)min(max(x, 0), d.nx - 1);
    Off off[R + 2];
#pragma unroll
    for (int j = 0; j < R + 2; ++j) off[j] = ((Off)min(max(y0 + j - 1, 0), d.ny - 1) * (Off)d.nx + xc) * 4;
    auto at = [](const float* p, Off b) { return __ldg(reinterpret_cast<const float*>(reinterpret_cast<const char*>(p) + b)); };
    auto put = [](float* p, Off b, float v) { *reinterpret_cast<float*>(reinterpret_cast<char*>(p) + b) = v; };
    struct Slice {
        float u[R + 1], pz[R + 1], py[R + 1], px[R + 1];   // u after the half step, p before it
    };
    // slice z at rows 0..R: p as read, u from it, from pz of slice z - 1 and from f
    auto form = [&](int z, const float (&below)[R + 1], Slice& S) {
        const size_t zo = (size_t)z * plane;
        float fv[R + 1], left = 0.f;
        // f: the image between its slice 1 and zeros (zeros on both sides of a single slice)
        if (z == 0 ? d.nzp > 3 : z < d.nzp - 1) {
            const float* sf = a.src + (z == 0 ? plane : zo - plane);
#pragma unroll
            for (int j = 0; j <= R; ++j) fv[j] = at(sf, off[j + 1]);
        } else {
#pragma unroll
            for (int j = 0; j <= R; ++j) fv[j] = 0.f;
        }
        if (FIRST) {
#pragma unroll
            for (int j = 0; j <= R; ++j) {
                S.u[j] = fv[j];
                S.pz[j] = S.py[j] = S.px[j] = 0.f;
            }
        } else {
            const float *u = a.u + zo, *pz = a.pz + zo, *py = a.py + zo, *px = a.px + zo;
#pragma unroll
            for (int j = 0; j <= R; ++j) {
                S.pz[j] = at(pz, off[j + 1]);
                S.py[j] = at(py, off[j + 1]);
                S.px[j] = at(px, off[j + 1]);
                S.u[j] = at(u, off[j + 1]);
            }
            left = at(py, off[0]);
        }
        const float below_y = y0 > 0 ? left : 0.f;
#pragma unroll
        for (int j = 0; j <= R; ++j) {
            float div = z > 0 ? (S.pz[j] - below[j]) * d.idz : S.pz[j];
            div += j ? (S.py[j] - S.py[j ? j - 1 : 0]) * d.idy : (S.py[0] - below_y) * sy0;
            const float l = __shfl_up_sync(0xffffffffu, S.px[j], 1);
            div += (S.px[j] - (x > 0 ? l : 0.f)) * sx;
            S.u[j] = S.u[j] * (1.f - a.tau1) + a.tau1 * (fv[j] + a.inv_lambda * div);
        }
    };
    // writes slice z from C with u of slice z + 1 from N (formed here)
    auto step = [&](int z, Slice& C, Slice& N) {
        if (LAST) {
            if (z >= 1 && z < d.nzp - 1 && out) {
                float* o = a.u_out + ((size_t)z * plane - plane);
#pragma unroll
                for (int j = 0; j < R; ++j)
                    if (y0 + j < d.ny) put(o, off[j + 1], C.u[j]);
            }
            if (z + 1 < zend) form(z + 1, C.pz, N);
            return;
        }
        const bool up = z + 1 < d.nzp;
        if (up) form(z + 1, C.pz, N);
        const float iz = up ? d.idz : 0.f;
        const size_t zo = (size_t)z * plane;
        float *ou = a.u_out + zo, *oz = a.pz_out + zo, *oy = a.py_out + zo, *ox = a.px_out + zo;
#pragma unroll
        for (int j = 0; j < R; ++j) {
            const float ux = __shfl_down_sync(0xffffffffu, C.u[j], 1);
            const float gz = (up ? N.u[j] - C.u[j] : 0.f) * iz;
            const float gy = y0 + j + 1 < d.ny ? (C.u[j + 1] - C.u[j]) * d.idy : 0.f;
            const float gx = ix != 0.f ? (ux - C.u[j]) * ix : 0.f;
            const float q0 = C.pz[j] + a.tau2 * gz, q1 = C.py[j] + a.tau2 * gy, q2 = C.px[j] + a.tau2 * gx;
            const float w = prox_shrink(q0 * q0 + q1 * q1 + q2 * q2);
            if (out && y0 + j < d.ny) {
                put(ou, off[j + 1], C.u[j]);
                put(oz, off[j + 1], q0 * w);
                put(oy, off[j + 1], q1 * w);
                put(ox, off[j + 1], q2 * w);
            }
        }
    };
    Slice A, B;
    {
        float below[R + 1];
#pragma unroll
        for (int j = 0; j <= R; ++j) below[j] = !FIRST && z0 > 0 ? at(a.pz + (size_t)(z0 - 1) * plane, off[j + 1]) : 0.f;
        form(z0, below, A);
    }
#pragma unroll 1
    for (int z = z0; z < zend; z += 2) {
        step(z, A, B);
        if (z + 1 >= zend) break;
        step(z + 1, B, A);
    }
}

int fused_denoise(const float* d_src, float* d_dst, const ProxDims& d, float lambda, int max_iter, float* d_work,
                  cudaStream_t st) {
    const size_t plane = (size_t)d.nx * d.ny, n = plane * d.nzp, nsrc = plane * (d.nzp - 2);
    float* w[8];
    for (int i = 0; i < 8; ++i) w[i] = d_work + (size_t)i * n;   // u, pz, py, px of each side
    if (max_iter == 0) {
        if (d_dst != d_src) TIGRE_CUDA(cudaMemcpyAsync(d_dst, d_src, sizeof(float) * nsrc, cudaMemcpyDeviceToDevice, st));
        return TIGRE_SUCCESS;
    }
    // the last pass reads the image while it writes the result: an overlapping result goes through u
    const uintptr_t s0 = (uintptr_t)d_src, t0 = (uintptr_t)d_dst, len = nsrc * sizeof(float);
    const bool overlap = s0 < t0 + len && t0 < s0 + len;
    const long tx = (d.nx + kStepLanes - 1) / kStepLanes, ty = (d.ny + kStepRows * kStepWarps - 1) / (kStepRows * kStepWarps);
    // slices per chunk: the fewest steps over the rounds of resident blocks (a chunk starts with a step)
    int zc = 0;
    long blocks = 0;
    double best = 0.0;
    for (int c = 2; c <= 128; c += c < 16 ? 1 : c / 8) {
        const long b = tx * ty * ((d.nzp + c - 1) / c);
        const double cost = (double)((b + 148 * kStepBlocks - 1) / (148 * kStepBlocks)) * (c + 1.0);
        if (zc == 0 || cost < best) { best = cost; zc = c; blocks = b; }
    }
    if (blocks > INT_MAX) return fail(TIGRE_ERR_BAD_ASSERT, "volume too large");
    float* result = overlap ? w[(max_iter & 1) ? 4 : 0] : d_dst;
    for (int i = 0; i < max_iter; ++i) {
        float** in = w + ((i & 1) ? 4 : 0);
        float** to = w + ((i & 1) ? 0 : 4);
        const float tau2 = 0.3f + 0.02f * (float)i;
        const float tau1 = (1.f / tau2) * ((1.f / 6.f) - (5.f / (15.f + (float)i)));
        const bool first = i == 0, last = i + 1 == max_iter;
        ProxStep a{d_src, in[0], in[1], in[2], in[3], last ? result : to[0], to[1], to[2], to[3], tau1, tau2,
                   1.f / lambda, zc};
        const unsigned grid = (unsigned)blocks;
        auto go = [&](auto off) {
            using Off = decltype(off);
            if (first && last) prox_step_kernel<true, true, Off><<<grid, 32 * kStepWarps, 0, st>>>(a, d);
            else if (first) prox_step_kernel<true, false, Off><<<grid, 32 * kStepWarps, 0, st>>>(a, d);
            else if (last) prox_step_kernel<false, true, Off><<<grid, 32 * kStepWarps, 0, st>>>(a, d);
            else prox_step_kernel<false, false, Off><<<grid, 32 * kStepWarps, 0, st>>>(a, d);
        };
        if (plane < 1000000000) go(0u);
        else go((size_t)0);
        TIGRE_LAUNCHED();
    }
    if (overlap) TIGRE_CUDA(cudaMemcpyAsync(d_dst, result, sizeof(float) * nsrc, cudaMemcpyDeviceToDevice, st));
    return TIGRE_SUCCESS;
}

}  // namespace
}  // namespace tigre

using namespace tigre;

extern "C" {

long long tigre_tv_denoise_work_floats(long nx, long ny, long nz) {
    return 5LL * nx * ny * (nz + 2);
}

long long tigre_tv_denoise_fused_floats(long nx, long ny, long nz) {
    return 8LL * nx * ny * (nz + 2);
}

int tigre_tv_denoise(const float* d_src, float* d_dst, long nx, long ny, long nz, float lambda, const float* spacing,
                     int max_iter, float* d_work, void* stream) {
    return tigre_tv_denoise_ex(d_src, d_dst, nx, ny, nz, lambda, spacing, max_iter, d_work,
                               tigre_tv_denoise_work_floats(nx, ny, nz), stream);
}

int tigre_tv_denoise_ex(const float* d_src, float* d_dst, long nx, long ny, long nz, float lambda,
                        const float* spacing, int max_iter, float* d_work, long long work_floats, void* stream) {
    TIGRE_NVTX("tigre_tv_denoise");
    if (!d_src || !d_dst || !d_work || nx <= 0 || ny <= 0 || nz <= 0 || max_iter < 0)
        return fail(TIGRE_ERR_BAD_ASSERT, "bad TV denoising arguments");
    if (!(lambda > 0.f)) return fail(TIGRE_ERR_BAD_ASSERT, "TV denoising: lambda must be positive");
    if ((double)nx * ny * (nz + 2) >= 9.0e18 / 5) return fail(TIGRE_ERR_BAD_ASSERT, "volume too large");
    const float sx = spacing ? spacing[0] : 1.f, sy = spacing ? spacing[1] : 1.f, sz = spacing ? spacing[2] : 1.f;
    if (!(sx > 0.f && sy > 0.f && sz > 0.f)) return fail(TIGRE_ERR_BAD_ASSERT, "TV denoising: spacing must be positive");
    if (work_floats < tigre_tv_denoise_work_floats(nx, ny, nz))
        return fail(TIGRE_ERR_BAD_ASSERT, "TV denoising: work space too small");
    cudaStream_t st = (cudaStream_t)stream;
    // a warp of the one-pass form takes four rows: of a single one three are idle (512 x 1 x 512, 6 iterations 88 us
    // against 78 in two passes)
    if (ny > 1 && work_floats >= tigre_tv_denoise_fused_floats(nx, ny, nz))
        return fused_denoise(d_src, d_dst, ProxDims{(int)nx, (int)ny, (int)(nz + 2), 1.f / sx, 1.f / sy, 1.f / sz},
                             lambda, max_iter, d_work, st);
    const long plane = nx * ny, n = plane * (nz + 2);
    float* f = d_work;
    float* u = f + n;
    float* pz = u + n;
    float* py = pz + n;
    float* px = py + n;
    // f: [image slice 1 | image | zeros] (zeros also for a single-slice image)
    TIGRE_CUDA(cudaMemsetAsync(f, 0, sizeof(float) * n, st));
    if (nz > 1) TIGRE_CUDA(cudaMemcpyAsync(f, d_src + plane, sizeof(float) * plane, cudaMemcpyDeviceToDevice, st));
    TIGRE_CUDA(cudaMemcpyAsync(f + plane, d_src, sizeof(float) * plane * nz, cudaMemcpyDeviceToDevice, st));
    TIGRE_CUDA(cudaMemcpyAsync(u, f, sizeof(float) * n, cudaMemcpyDeviceToDevice, st));
    TIGRE_CUDA(cudaMemsetAsync(pz, 0, sizeof(float) * n * 3, st));
    ProxDims d{(int)nx, (int)ny, (int)(nz + 2), 1.f / sx, 1.f / sy, 1.f / sz};
    const int grid = grid_for_prox(d);
    for (int i = 0; i < max_iter; ++i) {
        const float tau2 = 0.3f + 0.02f * (float)i;
        const float tau1 = (1.f / tau2) * ((1.f / 6.f) - (5.f / (15.f + (float)i)));
        prox_update_u<<<grid, 256, 0, st>>>(f, pz, py, px, u, tau1, 1.f / lambda, d);
        TIGRE_LAUNCHED();
        prox_update_p<<<grid, 256, 0, st>>>(u, pz, py, px, tau2, d);
        TIGRE_LAUNCHED();
    }
    TIGRE_CUDA(cudaMemcpyAsync(d_dst, u + plane, sizeof(float) * plane * nz, cudaMemcpyDeviceToDevice, st));
    return TIGRE_SUCCESS;
}

}  // extern "C"
