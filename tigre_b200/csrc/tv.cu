// POCS total-variation descent, sm_100a.
//
// One step of pocs_tv (Common/CUDA/GD_TV.cu:440-597) is
//     g = grad TV(f)                                  (gradientTV, :117-143)
//     f <- f - alpha * g / sqrt(sum(g^2) + 1e-7)      (:556-597)
// The reference runs gradientTV, a device copy, two reduction kernels, a host
// synchronisation and three element-wise kernels per step (~48 B/voxel).
// Here a step is two passes and no host round trip (~12 B/voxel):
//   pass 1  tv_march_kernel<kTvOutNorm>    stencil -> g, sum g^2 (FP64, one atomic per block)
//   pass 2  tv_march_kernel<kTvOutUpdate>  stencil again -> g, writes f - alpha g / |g|,
//                             reading |g|^2 from device memory (ping-pong buffers)
// g is recomputed rather than stored: the stencil is cheap, the bytes are not.
//
// Boundary rule of the single-device reference call: the image sits between
// zero slices in z (its zeroed halo buffer, GD_TV.cu:380-393 and 447-461);
// along x and y a difference whose neighbour is outside is 0 (gradient(), :91-115),
// and the terms of neighbours beyond the last x / y index vanish.

#include <cmath>
#include <cstdlib>
#include <mutex>
#include <string>

#include "tigre_internal.h"

namespace tigre {
namespace {

struct TVDims {
    int nx, ny, nz;
};

// Voxels (x, y, z < nzr) of the per-voxel kernels: blocks stride over (y, z) rows, threads over
// x, so no thread divides a linear index; i is the linear index of (x, y, z).
#define TV_FOR_EACH_VOXEL(d, nzr, x, y, z, i)                                                     \
    for (long row_ = blockIdx.x; row_ < (long)(d).ny * (nzr); row_ += gridDim.x) {               \
        const int y = (int)(row_ % (d).ny), z = (int)(row_ / (d).ny);                             \
        for (int x = threadIdx.x; x < (d).nx; x += blockDim.x) {                                   \
            const size_t i = ((size_t)z * (d).ny + y) * (d).nx + x;
#define TV_END_FOR_EACH_VOXEL \
    }                         \
    }

int grid_rows(const TVDims& d, int nzr) { return (int)std::min<long>((long)d.ny * nzr, 148 * 16); }

__device__ __forceinline__ float fget(const float* __restrict__ f, const TVDims& d, int x, int y, int z) {
    return (z >= 0 && z < d.nz) ? __ldg(f + ((size_t)z * d.ny + y) * d.nx + x) : 0.f;
}

__device__ __forceinline__ double block_sum(double v) {
    __shared__ double red[32];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    if (lane == 0) red[wid] = v;
    __syncthreads();
    v = 0.0;
    if (wid == 0) {
        const int nw = (blockDim.x + 31) >> 5;
        v = lane < nw ? red[lane] : 0.0;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
    }
    return v;
}

struct TVStep {
    const float* prior;   // PICCS prior image (same layout as f)
    float inv_delta;      // AwTV: 1 / delta
    float ratio;          // PICCS: weight of the prior term
    double norm_eps;      // added to sum(g^2) before the square root
    float grad_eps;       // added to every gradient norm: 1e-8 (GD_AwTV.cu:131), 1e-6 (PICCS.cu:149)
};

constexpr int kTvPocs = 0, kTvAw = 1, kTvPiccs = 2;

// ---- gradientTV in registers: POCS-TV, AwTV and PICCS passes and the autograd gradient ----
//
// At every point the backward differences (dz, dy, dx), their weighted forms (nz, ny, nx) and
// r = 1 / (sqrt(nz dz + ny dy + nx dx) + eps) -- unweighted for POCS-TV (gradientTV,
// GD_TV.cu:117-143), with w = exp(-(d / delta)^2) per component for AwTV (GD_AwTV.cu:117-158).
// The gradient at (x, y, z) (dftv, GD_TV.cu:135-140) is then
//     (nz + ny + nx) r  -  nx(x+1) r(x+1)  -  ny(y+1) r(y+1)  -  nz(z+1) r(z+1),
// each norm and weight evaluated once per voxel.  The differences are the reference's exactly;
// r uses the hardware reciprocal square root and reciprocal, so each term carries a relative
// error of a few 1e-7 against the reference's IEEE divisions.
// PICCS (PICCS.cu:117-154) runs on the bare image (no z difference at z = 0, no +z term at the
// last slice, eps 1e-6) with two fields, f and f - prior, for
// g = (1 - ratio) grad TV(f) + ratio grad TV(f - prior).
//
// A warp owns 30 x tv_rows(KIND) columns and marches down a chunk of slices with everything in
// registers: each lane holds one x of rows y0-1 .. y0+R of the previous and the current slice
// (the next one is being fetched), the x neighbours come by shuffle (lanes 0 and 31 only
// supply them), the y ones are the lane's own rows, and the +z term completes a slice one
// step later.  No shared memory and no barrier.  Coordinates outside the volume are clamped when
// loading, which makes the differences across the -x / -y faces and the terms beyond the last
// x / y index exactly 0; the zero slices below z = 0 and above z = nz - 1 (POCS-TV, AwTV) are
// staged as zeros, and PICCS repeats its end slices there.
//
// Bound by instruction issue (256^3: 46 thread instructions per voxel at 66-69 % of the issue slots,
// beyond the arithmetic the three shuffles, the addresses and the rows shared with the
// neighbouring warp), on small volumes by the latency of the few steps.  Per step of two passes:
// 512^3 473 us (shared-memory tiles with one barrier per slice: 1113), 301 x 333 x 317 123 us (272),
// 64^3 14 us (58).  4, 6 or 8 rows per warp with 8, 6 or 5 blocks per SM: 481 / 484 / 497 us at 512^3.
constexpr int kTvLanes = 30;   // output columns of a warp
constexpr int kTvWarps = 4;    // warps of a block, neighbours in y (they share their edge rows in L1)
constexpr int kTvOutNorm = 0, kTvOutUpdate = 1, kTvOutGrad = 2;

// rows of a warp's tile.  PICCS, with two fields in registers, takes fewer.
constexpr int tv_rows(int kind) { return kind == kTvPiccs ? 4 : 6; }
constexpr int tv_blocks(int kind) { return kind == kTvPiccs ? 5 : 6; }   // resident blocks per SM that registers allow

struct TvTiles {
    int tx, ty, zc;   // tiles in x and (block) tiles in y, slices per chunk
    unsigned blocks;
};

// Slices per chunk: the fewest steps over the rounds of resident blocks, a chunk of zc slices
// taking zc + 1 steps and about half a step to start.
TvTiles tv_tiles(const TVDims& d, int kind) {
    const int span = tv_rows(kind) * kTvWarps;
    const int tx = (d.nx + kTvLanes - 1) / kTvLanes, ty = (d.ny + span - 1) / span;
    const long slots = 148L * tv_blocks(kind);
    TvTiles t{tx, ty, 0, 0};
    double best = 0.0;
    for (int zc = 2; zc <= 128; zc += zc < 16 ? 1 : zc / 8) {
        const long blocks = (long)tx * ty * ((d.nz + zc - 1) / zc);
        const double cost = (double)((blocks + slots - 1) / slots) * (zc + 1.5);
        if (t.zc == 0 || cost < best) { best = cost; t.zc = zc; t.blocks = (unsigned)blocks; }
    }
    return t;
}

__device__ __forceinline__ float tv_rsqrt(float a) {
    float r;
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(a));
    return r;
}
__device__ __forceinline__ float tv_rcp(float a) {
    float r;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(a));
    return r;
}

// 1 / (sqrt(s) + eps) for the squared norm s = wz dz + wy dy + wx dx >= 0.  The smallest normal
// number in the sum keeps the reciprocal square root finite at s = 0; it changes no value of
// r, since a root below 1e-15 vanishes beside eps.
__device__ __forceinline__ float tv_rnorm(float wz, float wy, float wx, float dz, float dy, float dx, float eps) {
    const float s = fmaf(wx, dx, fmaf(wz, dz, fmaf(wy, dy, 1.1754944e-38f)));
    return tv_rcp(__fadd_rn(__fmul_rn(s, tv_rsqrt(s)), eps));
}

// OUT: kTvOutNorm adds sum g^2 (FP64, one atomic per block) into *sums; kTvOutUpdate writes
// o = f - alpha g / sqrt(*sums + st.norm_eps) (GD_TV.cu:556-597); kTvOutGrad writes o = g.
// KIND: kTvPocs, kTvAw or kTvPiccs.  Off: type of the byte offsets within a slice (32 bits wherever a
// slice is below 4 GB, so that a load is one instruction on the slice's uniform base).
template <int OUT, int KIND, typename Off>
__global__ void __launch_bounds__(32 * kTvWarps, tv_blocks(KIND)) tv_march_kernel(const float* __restrict__ f,
                                                                           float* __restrict__ o, TVDims d, TvTiles T,
                                                                           TVStep st, double* __restrict__ sums,
                                                                           float alpha) {
    constexpr bool HALO = KIND != kTvPiccs;
    constexpr int NF = KIND == kTvPiccs ? 2 : 1;   // fields: f (and f - prior)
    constexpr int R = tv_rows(KIND);
    const int lane = threadIdx.x & 31, wid = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0);
    const int bx = (int)(blockIdx.x % (unsigned)T.tx), bt = (int)(blockIdx.x / (unsigned)T.tx);
    const int x = bx * kTvLanes + lane - 1, y0 = (bt % T.ty * kTvWarps + wid) * R;
    const int z0 = bt / T.ty * T.zc, zend = min(z0 + T.zc, d.nz);   // slice zend supplies the +z term
    const size_t plane = (size_t)d.nx * d.ny;
    const float eps = st.grad_eps, idl = st.inv_delta;
    float scale = 0.f;
    if (OUT == kTvOutUpdate) scale = (float)((double)alpha / sqrt(*sums + st.norm_eps));
    double acc = 0.0;
    const int nrow = lane >= 1 && lane <= kTvLanes && x < d.nx ? min(R, d.ny - y0) : 0;   // rows this lane writes
    // byte offsets in a slice of the rows y0-1 .. y0+R, clamped to the volume
    const Off xc = (Off)min(max(x, 0), d.nx - 1);
    Off off[R + 2];
#pragma unroll
    for (int j = 0; j < R + 2; ++j) off[j] = ((Off)min(max(y0 + j - 1, 0), d.ny - 1) * (Off)d.nx + xc) * 4;
    auto at = [](const float* p, Off b) { return __ldg(reinterpret_cast<const float*>(reinterpret_cast<const char*>(p) + b)); };
    auto fetch = [&](int z, float (&v)[NF][R + 2]) {
        if (HALO) {
            if (z >= 0 && z < d.nz) {
                const float* p = f + (size_t)z * plane;
#pragma unroll
                for (int j = 0; j < R + 2; ++j) v[0][j] = at(p, off[j]);
            } else {
#pragma unroll
                for (int j = 0; j < R + 2; ++j) v[0][j] = 0.f;
            }
        } else {
            const size_t zl = (size_t)min(max(z, 0), d.nz - 1) * plane;
            const float *p = f + zl, *q = st.prior + zl;
#pragma unroll
            for (int j = 0; j < R + 2; ++j) {
                v[0][j] = at(p, off[j]);
                v[NF - 1][j] = v[0][j] - at(q, off[j]);
            }
        }
    };
    float part[NF][R];
    // slice z: P, C and N hold slices z - 1, z and z + 1 (being fetched)
    auto step = [&](int z, float (&P)[NF][R + 2], float (&C)[NF][R + 2], float (&N)[NF][R + 2]) {
        if (z < zend) fetch(z + 1, N);
        const int emit = z > z0 ? nrow : 0;   // rows of slice z - 1, complete with its +z neighbour's term
        char* ob = OUT == kTvOutNorm ? nullptr : reinterpret_cast<char*>(o + ((size_t)z * plane - plane));
#pragma unroll
        for (int j = 0; j <= R; ++j) {   // points of row y0 + j
            float gc[NF];
#pragma unroll
            for (int c = 0; c < NF; ++c) {
                const float v = C[c][j + 1];
                const float dz = v - P[c][j + 1], dy = v - C[c][j];
                const float dx = v - __shfl_up_sync(0xffffffffu, v, 1);
                float wz = dz, wy = dy, wx = dx;
                if (KIND == kTvAw) {
                    const float tz = dz * idl, ty = dy * idl, tx = dx * idl;
                    wz = expf(-(tz * tz)) * dz;
                    wy = expf(-(ty * ty)) * dy;
                    wx = expf(-(tx * tx)) * dx;
                }
                const float r = tv_rnorm(wz, wy, wx, dz, dy, dx, eps);
                if (j > 0) part[c][j - 1] = fmaf(-wy, r, part[c][j - 1]);   // the +y term of the row below
                if (j < R) {
                    const float rx = __shfl_down_sync(0xffffffffu, r, 1), wx1 = __shfl_down_sync(0xffffffffu, wx, 1);
                    gc[c] = fmaf(-wz, r, part[c][j]);
                    part[c][j] = fmaf(-wx1, rx, (wz + wy + wx) * r);
                }
            }
            if (j == R) break;
            if (j < emit) {
                const float g = NF == 2 ? fmaf(1.f - st.ratio, gc[0], st.ratio * gc[NF - 1]) : gc[0];
                if (OUT == kTvOutNorm) acc = fma((double)g, (double)g, acc);
                else *reinterpret_cast<float*>(ob + off[j + 1]) = OUT == kTvOutUpdate ? fmaf(-scale, g, P[0][j + 1]) : g;
            }
        }
    };
    if (y0 < d.ny) {
        float A[NF][R + 2], B[NF][R + 2], C[NF][R + 2];
        fetch(z0 - 1, A);
        fetch(z0, B);
#pragma unroll
        for (int c = 0; c < NF; ++c)
#pragma unroll
            for (int j = 0; j < R; ++j) part[c][j] = 0.f;
        // three steps bring the register sets back to their starting roles
        for (int z = z0; z <= zend; z += 3) {
            step(z, A, B, C);
            if (z + 1 > zend) break;
            step(z + 1, B, C, A);
            if (z + 2 > zend) break;
            step(z + 2, C, A, B);
        }
    }
    if (OUT == kTvOutNorm) {
        acc = block_sum(acc);
        if (threadIdx.x == 0) atomicAdd(sums, acc);
    }
}

template <int OUT, int KIND>
void launch_tv(const float* f, float* o, const TVDims& d, const TVStep& st, double* sums, float alpha, cudaStream_t s) {
    const TvTiles T = tv_tiles(d, KIND);
    if ((double)d.nx * d.ny < 1.0e9)
        tv_march_kernel<OUT, KIND, unsigned><<<T.blocks, 32 * kTvWarps, 0, s>>>(f, o, d, T, st, sums, alpha);
    else
        tv_march_kernel<OUT, KIND, size_t><<<T.blocks, 32 * kTvWarps, 0, s>>>(f, o, d, T, st, sums, alpha);
}

// POCS-TV step parameters (GD_TV.cu): no prior, no weights, 1e-7 under the norm, 1e-8 per gradient
constexpr TVStep kPocsStep{nullptr, 0.f, 0.f, 1e-7, 1e-8f};

// sum_i |grad f_i| over the voxels and the zero halo slice above the last one
// (whose gradient norm is |f(x,y,nz-1)|); its derivative is the gradient of tv_march_kernel.
__global__ void __launch_bounds__(256) tv_value_kernel(const float* __restrict__ f, TVDims d, double* __restrict__ out) {
    double s = 0.0;
    TV_FOR_EACH_VOXEL(d, d.nz + 1, x, y, z, i) {
        (void)i;
        if (z == d.nz) {
            s += fabs((double)fget(f, d, x, y, z - 1));
            continue;
        }
        const float c = fget(f, d, x, y, z);
        const float d0 = c - fget(f, d, x, y, z - 1);
        const float d1 = y > 0 ? c - fget(f, d, x, y - 1, z) : 0.f;
        const float d2 = x > 0 ? c - fget(f, d, x - 1, y, z) : 0.f;
        s += sqrt((double)d0 * d0 + (double)d1 * d1 + (double)d2 * d2);
    }
    TV_END_FOR_EACH_VOXEL
    s = block_sum(s);
    if (threadIdx.x == 0) atomicAdd(out, s);
}

}  // namespace
}  // namespace tigre

using namespace tigre;

extern "C" {

int tigre_tv_gradient(const void* d_img, int dtype, float* d_grad, long nx, long ny, long nz, void* stream) {
    if (dtype != TIGRE_F32) return fail(TIGRE_ERR_BAD_ASSERT, "TV kernels take float32 volumes");
    if (nx <= 0 || ny <= 0 || nz <= 0 || !d_img || !d_grad) return fail(TIGRE_ERR_BAD_ASSERT, "bad TV arguments");
    TVDims d{(int)nx, (int)ny, (int)nz};
    launch_tv<kTvOutGrad, kTvPocs>((const float*)d_img, d_grad, d, kPocsStep, nullptr, 0.f, (cudaStream_t)stream);
    TIGRE_LAUNCHED();
    return TIGRE_SUCCESS;
}

int tigre_tv_value(const void* d_img, int dtype, long nx, long ny, long nz, double* d_out, void* stream) {
    if (dtype != TIGRE_F32) return fail(TIGRE_ERR_BAD_ASSERT, "TV kernels take float32 volumes");
    if (nx <= 0 || ny <= 0 || nz <= 0 || !d_img || !d_out) return fail(TIGRE_ERR_BAD_ASSERT, "bad TV arguments");
    TVDims d{(int)nx, (int)ny, (int)nz};
    tv_value_kernel<<<grid_rows(d, d.nz + 1), 256, 0, (cudaStream_t)stream>>>((const float*)d_img, d, d_out);
    TIGRE_LAUNCHED();
    return TIGRE_SUCCESS;
}

// In-place POCS-TV.  d_work: nx*ny*nz floats of caller scratch; 8 bytes of
// reduction scratch are taken from the stream-ordered allocator.
int tigre_tv_pocs(void* d_img, int dtype, long nx, long ny, long nz, float alpha, int max_iter, float* d_work,
                  void* stream) {
    TIGRE_NVTX("tigre_tv_pocs");
    if (dtype != TIGRE_F32) return fail(TIGRE_ERR_BAD_ASSERT, "TV kernels take float32 volumes");
    if (nx <= 0 || ny <= 0 || nz <= 0 || !d_img || !d_work || max_iter < 0)
        return fail(TIGRE_ERR_BAD_ASSERT, "bad TV arguments");
    if ((double)nx * ny * nz >= 2147483647.0) return fail(TIGRE_ERR_BAD_ASSERT, "volume too large");
    cudaStream_t st = (cudaStream_t)stream;
    TVDims d{(int)nx, (int)ny, (int)nz};
    const size_t n = (size_t)nx * ny * nz;
    double* sums = nullptr;
    TIGRE_CUDA(cudaMallocAsync(&sums, sizeof(double) * (size_t)std::max(max_iter, 1), st));
    TIGRE_CUDA(cudaMemsetAsync(sums, 0, sizeof(double) * (size_t)std::max(max_iter, 1), st));
    float* cur = (float*)d_img;
    float* nxt = d_work;
    for (int it = 0; it < max_iter; ++it) {
        launch_tv<kTvOutNorm, kTvPocs>(cur, nullptr, d, kPocsStep, sums + it, 0.f, st);
        launch_tv<kTvOutUpdate, kTvPocs>(cur, nxt, d, kPocsStep, sums + it, alpha, st);
        std::swap(cur, nxt);
    }
    if (cur != (float*)d_img) TIGRE_CUDA(cudaMemcpyAsync(d_img, cur, n * sizeof(float), cudaMemcpyDeviceToDevice, st));
    TIGRE_CUDA(cudaFreeAsync(sums, st));
    TIGRE_CUDA(cudaGetLastError());
    note_launches(2ull * (unsigned long long)max_iter);
    return TIGRE_SUCCESS;
}

}  // extern "C"

// Shared driver of the weighted / prior TV descents: ping-pong between d_img and d_work.
template <int KIND>
static int tv_descent(void* d_img, long nx, long ny, long nz, float alpha, int max_iter, const TVStep& stp,
                      float* d_work, cudaStream_t st) {
    TVDims d{(int)nx, (int)ny, (int)nz};
    const size_t n = (size_t)nx * ny * nz;
    double* sums = nullptr;
    TIGRE_CUDA(cudaMallocAsync(&sums, sizeof(double) * (size_t)std::max(max_iter, 1), st));
    TIGRE_CUDA(cudaMemsetAsync(sums, 0, sizeof(double) * (size_t)std::max(max_iter, 1), st));
    float* cur = (float*)d_img;
    float* nxt = d_work;
    for (int it = 0; it < max_iter; ++it) {
        launch_tv<kTvOutNorm, KIND>(cur, nullptr, d, stp, sums + it, 0.f, st);
        launch_tv<kTvOutUpdate, KIND>(cur, nxt, d, stp, sums + it, alpha, st);
        std::swap(cur, nxt);
    }
    if (cur != (float*)d_img) TIGRE_CUDA(cudaMemcpyAsync(d_img, cur, n * sizeof(float), cudaMemcpyDeviceToDevice, st));
    TIGRE_CUDA(cudaFreeAsync(sums, st));
    TIGRE_CUDA(cudaGetLastError());
    note_launches(2ull * (unsigned long long)max_iter);
    return TIGRE_SUCCESS;
}

extern "C" {

// In-place adaptive-weighted TV descent (aw_pocs_tv, GD_AwTV.cu:276-720): per step
//   g = grad AwTV(f);  f <- f - alpha g / sqrt(sum g^2 + 1e-7).
int tigre_tv_aw_pocs(void* d_img, int dtype, long nx, long ny, long nz, float alpha, int max_iter, float delta,
                    float* d_work, void* stream) {
    TIGRE_NVTX("tigre_tv_aw_pocs");
    if (dtype != TIGRE_F32) return fail(TIGRE_ERR_BAD_ASSERT, "TV kernels take float32 volumes");
    if (nx <= 0 || ny <= 0 || nz <= 0 || !d_img || !d_work || max_iter < 0)
        return fail(TIGRE_ERR_BAD_ASSERT, "bad TV arguments");
    if ((double)nx * ny * nz >= 2147483647.0) return fail(TIGRE_ERR_BAD_ASSERT, "volume too large");
    if (!(delta != 0.f) || !std::isfinite(delta)) return fail(TIGRE_ERR_BAD_ASSERT, "AwTV: delta must be finite and nonzero");
    const TVStep stp{nullptr, 1.f / delta, 0.f, 1e-7, 1e-8f};
    return tv_descent<kTvAw>(d_img, nx, ny, nz, alpha, max_iter, stp, d_work, (cudaStream_t)stream);
}

// In-place PICCS TV descent (piccs_tv, PICCS.cu:274-380): per step
//   g = (1 - ratio) grad TV(f) + ratio grad TV(f - prior);  f <- f - alpha g / sqrt(sum g^2).
int tigre_tv_piccs(void* d_img, const void* d_prior, int dtype, long nx, long ny, long nz, float alpha, float ratio,
                   int max_iter, float* d_work, void* stream) {
    TIGRE_NVTX("tigre_tv_piccs");
    if (dtype != TIGRE_F32) return fail(TIGRE_ERR_BAD_ASSERT, "TV kernels take float32 volumes");
    if (nx <= 0 || ny <= 0 || nz <= 0 || !d_img || !d_prior || !d_work || max_iter < 0)
        return fail(TIGRE_ERR_BAD_ASSERT, "bad TV arguments");
    if ((double)nx * ny * nz >= 2147483647.0) return fail(TIGRE_ERR_BAD_ASSERT, "volume too large");
    const TVStep stp{(const float*)d_prior, 0.f, ratio, 0.0, 1e-6f};
    return tv_descent<kTvPiccs>(d_img, nx, ny, nz, alpha, max_iter, stp, d_work, (cudaStream_t)stream);
}

}  // extern "C"

// POCS-TV that allocates nothing.
//
// Who needs it: a caller whose process has handed all free device memory to another
// allocator (a framework's caching pool, a service run under a fixed memory cap) gets
// no memory from cudaMallocAsync, and a caller inside a fixed-latency loop must not
// enter the allocator at all, since allocation can block on locks or on the device.
// For those callers the only scratch of tigre_tv_pocs besides d_work -- one FP64 norm
// sum per iteration -- lives here in a fixed array of this module's device memory.
//
// Limits and sharing: the array holds kTvPocsStaticMaxIter sums, so max_iter above it
// is rejected.  Every call on a device uses the same array, and the first max_iter
// entries must be zero when a call's first kernel runs: each call clears them on its
// stream before use.  Calls that overlap in time on one device (other streams, other
// host threads) therefore race on the sums and must be serialised by the caller.
// The first call on each device looks up the array's address with that device
// current and caches it; make that first call before any stream capture.  A device
// reset invalidates the cached address: tigre_release_cache() forgets it, and the
// next call looks it up again.
constexpr int kTvPocsStaticMaxIter = 4096;   // 32 KiB
static __device__ __align__(256) double g_tv_pocs_sums[kTvPocsStaticMaxIter];

namespace {
constexpr int kMaxDevices = 256;
std::mutex g_tv_pocs_sums_mu;
double* g_tv_pocs_sums_addr[kMaxDevices] = {};

// Address of g_tv_pocs_sums on the current device (looked up once per device).
int tv_pocs_static_sums(double** out) {
    int dev = 0;
    TIGRE_CUDA(cudaGetDevice(&dev));
    if (dev < 0 || dev >= kMaxDevices) return fail(TIGRE_ERR_BAD_ASSERT, "device index out of range");
    std::lock_guard<std::mutex> lk(g_tv_pocs_sums_mu);
    if (!g_tv_pocs_sums_addr[dev]) {
        void* p = nullptr;
        const cudaError_t e = cudaGetSymbolAddress(&p, g_tv_pocs_sums);
        if (e != cudaSuccess || !p) return cuda_fail(e, "cudaGetSymbolAddress(g_tv_pocs_sums)");
        g_tv_pocs_sums_addr[dev] = (double*)p;
    }
    *out = g_tv_pocs_sums_addr[dev];
    return TIGRE_SUCCESS;
}
}  // namespace

namespace tigre {
void forget_static_addresses() {
    std::lock_guard<std::mutex> lk(g_tv_pocs_sums_mu);
    for (auto& a : g_tv_pocs_sums_addr) a = nullptr;
}
}  // namespace tigre

extern "C" int tigre_tv_pocs_noalloc(void* d_img, int dtype, long nx, long ny, long nz, float alpha, int max_iter,
                                     float* d_work, void* stream) {
    if (dtype != TIGRE_F32) return fail(TIGRE_ERR_BAD_ASSERT, "TV kernels take float32 volumes");
    if (nx <= 0 || ny <= 0 || nz <= 0 || !d_img || !d_work || max_iter < 0)
        return fail(TIGRE_ERR_BAD_ASSERT, "bad TV arguments");
    if ((double)nx * ny * nz >= 2147483647.0) return fail(TIGRE_ERR_BAD_ASSERT, "volume too large");
    if (max_iter > kTvPocsStaticMaxIter)
        return fail(TIGRE_ERR_BAD_ASSERT, "tigre_tv_pocs_noalloc: max_iter " + std::to_string(max_iter) +
                                              " exceeds its fixed scratch of " +
                                              std::to_string(kTvPocsStaticMaxIter) + " iterations");
    double* sums = nullptr;
    if (int rc = tv_pocs_static_sums(&sums)) return rc;
    cudaStream_t st = (cudaStream_t)stream;
    TVDims d{(int)nx, (int)ny, (int)nz};
    const size_t n = (size_t)nx * ny * nz;
    if (max_iter > 0) TIGRE_CUDA(cudaMemsetAsync(sums, 0, sizeof(double) * (size_t)max_iter, st));
    float* cur = (float*)d_img;
    float* nxt = d_work;
    for (int it = 0; it < max_iter; ++it) {
        launch_tv<kTvOutNorm, kTvPocs>(cur, nullptr, d, kPocsStep, sums + it, 0.f, st);
        launch_tv<kTvOutUpdate, kTvPocs>(cur, nxt, d, kPocsStep, sums + it, alpha, st);
        std::swap(cur, nxt);
    }
    if (cur != (float*)d_img) TIGRE_CUDA(cudaMemcpyAsync(d_img, cur, n * sizeof(float), cudaMemcpyDeviceToDevice, st));
    TIGRE_CUDA(cudaGetLastError());
    note_launches(2ull * (unsigned long long)max_iter);
    return TIGRE_SUCCESS;
}
