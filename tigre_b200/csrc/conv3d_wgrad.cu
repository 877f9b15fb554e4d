// Weight gradient of the 3x3x3 convolutions (sm_100a):
//
//   dw[co][t][ci] += sum_v dy[v][co] x[v + off(t)][ci]     (x 0 outside the volume)
//
// for BF16 channels-last x and dy, FP32 accumulation.  Written out as a GEMM over an im2col matrix
// this moves 27 copies of x through HBM (64^3 x 32 channels: 450 MB written and read, 2.25 ms of
// the 2.47 ms of a training step of the layer).  Here a block owns CO x 16 channels of all 27 taps
// and walks over voxel tiles of 16 x 4 x 4; a tile's x (with its one-voxel halo) and dy are staged
// once in shared memory by 16-byte cp.async copies, two tiles in flight, and the 27 taps read
// them at shifted rows.  Both operands are voxel-major, so the warp-level tensor-core fragments
// (m16n8k16, K = 16 voxels along x) come through ldmatrix.trans; rows are padded by 16 bytes,
// which makes the eight rows of a matrix fall in distinct banks.  Warp w of nine holds the three
// taps (dz, dy) = (w / 3, w % 3), dx = 0..2: the dy fragments of a step serve all three.  The
// tcgen05 form would pad 16- and 32-channel operands to 64 rows and needs 27 accumulator
// tiles, more columns than tensor memory has; at these widths the warp-level path is not the limit.
// 64^3, 32 -> 32 channels: 14.5 GFLOP in 57 us (254 TFLOP/s) and 6 us to add the slices; im2col took
// 1506 us and the GEMM 748 us.  The ReLU mask, the bias sums and the BF16 copy of the gradient are one
// pass of 14 us (five torch kernels, 100 us).
//
// The tiles are divided over `splits` blocks per channel tile, each writing its own slice of the
// partial sums, added up in a fixed order afterwards (no atomics).

#include <cuda_bf16.h>

#include <algorithm>

#include "tigre_internal.h"

namespace tigre {
namespace {

constexpr int kTX = 16, kTY = 4, kTZ = 4;                   // voxel tile
constexpr int kHX = kTX + 2, kHY = kTY + 2, kHZ = kTZ + 2;  // with halo
constexpr int kCI = 16;                                     // input channels per block
constexpr int kWgThreads = 9 * 32;
constexpr int kRowX = kCI * 2 + 16;                         // bytes of a staged voxel row of x
constexpr int kXBytes = kHX * kHY * kHZ * kRowX;

constexpr int row_dy(int co) { return co * 2 + 16; }
constexpr int stage_bytes(int co) { return kXBytes + kTX * kTY * kTZ * row_dy(co); }

struct WgArgs {
    const __nv_bfloat16* x;
    const __nv_bfloat16* dy;
    float* ws;               // [splits][Cout][27 Cin]
    int D, H, W, Cin, Cout;
    int tx, ty;
    long ntiles;
    int splits, nci;
};

__device__ __forceinline__ void cp16(uint32_t dst, const void* src, bool ok) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(dst), "l"(src), "r"(ok ? 16 : 0));
}

__device__ __forceinline__ void ldsm4t(uint32_t a, uint32_t (&r)[4]) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
                 : "r"(a)
                 : "memory");
}

__device__ __forceinline__ void mma(float (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
    asm volatile(
        "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
        : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
        : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

template <int CO>
__global__ void __launch_bounds__(kWgThreads, 2) conv_wgrad_kernel(WgArgs p) {
    constexpr int MT = CO / 16, kRowD = row_dy(CO), kStage = stage_bytes(CO);
    extern __shared__ __align__(128) unsigned char wg_smem[];
    const uint32_t base = (uint32_t)__cvta_generic_to_shared(wg_smem);
    const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
    const int ci0 = (int)(blockIdx.y % p.nci) * kCI, co0 = (int)(blockIdx.y / p.nci) * CO;
    auto load = [&](long tile, int buf) {
        const int bx = (int)(tile % p.tx);
        const long r = tile / p.tx;
        const int x0 = bx * kTX, y0 = (int)(r % p.ty) * kTY, z0 = (int)(r / p.ty) * kTZ;
        const uint32_t sx = base + (uint32_t)buf * kStage, sd = sx + kXBytes;
        for (int e = tid; e < kHX * kHY * kHZ * (kCI / 8); e += kWgThreads) {
            const int ch = e % (kCI / 8), v = e / (kCI / 8);
            const int hx = v % kHX, hy = v / kHX % kHY, hz = v / (kHX * kHY);
            const int gx = x0 + hx - 1, gy = y0 + hy - 1, gz = z0 + hz - 1;
            const bool ok = gx >= 0 && gx < p.W && gy >= 0 && gy < p.H && gz >= 0 && gz < p.D;
            const __nv_bfloat16* src = ok ? p.x + (((long)gz * p.H + gy) * p.W + gx) * p.Cin + ci0 + ch * 8 : p.x;
            cp16(sx + (uint32_t)(v * kRowX + ch * 16), src, ok);
        }
        for (int e = tid; e < kTX * kTY * kTZ * (CO / 8); e += kWgThreads) {
            const int ch = e % (CO / 8), v = e / (CO / 8);
            const int gx = x0 + v % kTX, gy = y0 + v / kTX % kTY, gz = z0 + v / (kTX * kTY);
            const bool ok = gx < p.W && gy < p.H && gz < p.D;
            const __nv_bfloat16* src = ok ? p.dy + (((long)gz * p.H + gy) * p.W + gx) * p.Cout + co0 + ch * 8 : p.dy;
            cp16(sd + (uint32_t)(v * kRowD + ch * 16), src, ok);
        }
        asm volatile("cp.async.commit_group;\n" ::);
    };
    float acc[3][MT][2][4];
#pragma unroll
    for (int t = 0; t < 3; ++t)
#pragma unroll
        for (int m = 0; m < MT; ++m)
#pragma unroll
            for (int n = 0; n < 2; ++n)
#pragma unroll
                for (int k = 0; k < 4; ++k) acc[t][m][n][k] = 0.f;
    const int tz = wid / 3, ty = wid % 3;
    // ldmatrix row addresses of this lane: A (dy): matrices (co 0-7, v 0-7), (co 8-15, v 0-7), (co 0-7, v 8-15),
    // (co 8-15, v 8-15); B (x): (v 0-7, ci 0-7), (v 8-15, ci 0-7), (v 0-7, ci 8-15), (v 8-15, ci 8-15)
    const uint32_t a_lane = (uint32_t)(((lane & 7) + (lane >> 4) * 8) * kRowD + ((lane >> 3) & 1) * 16);
    const uint32_t b_lane = (uint32_t)(((lane & 7) + ((lane >> 3) & 1) * 8) * kRowX + (lane >> 4) * 16);
    long tile = blockIdx.x;
    if (tile < p.ntiles) load(tile, 0);
    int buf = 0;
    for (; tile < p.ntiles; tile += p.splits, buf ^= 1) {
        const long next = tile + p.splits;
        if (next < p.ntiles) {
            load(next, buf ^ 1);
            asm volatile("cp.async.wait_group 1;\n" ::);
        } else {
            asm volatile("cp.async.wait_group 0;\n" ::);
        }
        __syncthreads();
        const uint32_t sx = base + (uint32_t)buf * kStage, sd = sx + kXBytes;
        // Places of the tile past the volume's end hold dy = 0, but x may have a voxel of the volume
        // beside them, and 0 times an infinite one is no 0: rows of such places are left out, and in the
        // others their x is cleared (K index 2 (lane % 4) + e of the low half, + 8 of the high one).
        const long tr = tile / p.tx;
        const int nx = p.W - (int)(tile % p.tx) * kTX, ny = min(p.H - (int)(tr % p.ty) * kTY, kTY);
        const int nz = min(p.D - (int)(tr / p.ty) * kTZ, kTZ);
        const int kx = (lane & 3) * 2;
        const uint32_t m0 = (kx < nx ? 0xffffu : 0u) | (kx + 1 < nx ? 0xffff0000u : 0u);
        const uint32_t m1 = (kx + 8 < nx ? 0xffffu : 0u) | (kx + 9 < nx ? 0xffff0000u : 0u);
#pragma unroll 1
        for (int z = 0; z < nz; ++z) {
#pragma unroll
            for (int y = 0; y < kTY; ++y) {
                if (y >= ny) break;
                uint32_t a[MT][4];
#pragma unroll
                for (int m = 0; m < MT; ++m)
                    ldsm4t(sd + (uint32_t)((z * kTY + y) * kTX * kRowD + m * 32) + a_lane, a[m]);
                const uint32_t row = sx + (uint32_t)(((z + tz) * kHY + y + ty) * kHX * kRowX) + b_lane;
#pragma unroll
                for (int t = 0; t < 3; ++t) {
                    uint32_t b[4];
                    ldsm4t(row + (uint32_t)(t * kRowX), b);
                    b[0] &= m0;
                    b[1] &= m1;
                    b[2] &= m0;
                    b[3] &= m1;
#pragma unroll
                    for (int m = 0; m < MT; ++m) {
                        mma(acc[t][m][0], a[m], b[0], b[1]);
                        mma(acc[t][m][1], a[m], b[2], b[3]);
                    }
                }
            }
        }
        __syncthreads();   // the next iteration's copy refills this buffer
    }
    float* o = p.ws + (size_t)blockIdx.x * p.Cout * 27 * p.Cin;
#pragma unroll
    for (int t = 0; t < 3; ++t)
#pragma unroll
        for (int m = 0; m < MT; ++m)
#pragma unroll
            for (int n = 0; n < 2; ++n)
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    const int co = co0 + 16 * m + (lane >> 2) + 8 * h, ci = ci0 + 8 * n + (lane & 3) * 2;
                    float* q = o + ((size_t)co * 27 + 9 * tz + 3 * ty + t) * p.Cin + ci;
                    *reinterpret_cast<float2*>(q) = make_float2(acc[t][m][n][2 * h], acc[t][m][n][2 * h + 1]);
                }
}

// dst[i] += sum over s < splits of ws[s * n + i], in order of s
__global__ void __launch_bounds__(256) wgrad_reduce_kernel(const float* __restrict__ ws, float* __restrict__ dst, long n,
                                                           int splits) {
    const long i = blockIdx.x * (long)blockDim.x + threadIdx.x;
    if (i >= n) return;
    float acc = dst[i];
    int s = 0;
    for (; s + 8 <= splits; s += 8) {
        float v[8];
#pragma unroll
        for (int k = 0; k < 8; ++k) v[k] = __ldg(ws + (s + k) * n + i);
#pragma unroll
        for (int k = 0; k < 8; ++k) acc += v[k];
    }
    for (; s < splits; ++s) acc += __ldg(ws + s * n + i);
    dst[i] = acc;
}

// g = dy (y > 0), and per block the sums of g over its voxels, by channel: the ReLU's and the
// bias's share of a convolution's backward pass.  A thread keeps one group of eight channels
// (the stride is a multiple of the groups); partial[block][C] is added up in order afterwards.
__global__ void __launch_bounds__(256) relu_grad_kernel(const uint4* __restrict__ dy, const uint4* __restrict__ y,
                                                        uint4* __restrict__ g, float* __restrict__ partial, long nvec,
                                                        int groups, int relu) {
    extern __shared__ float rg_sums[];   // [threads][8]
    const int per = blockDim.x / groups * groups;   // threads that work: a multiple of the groups
    float s[8] = {};
    if ((int)threadIdx.x < per) {
        const long stride = (long)gridDim.x * per;
        for (long i = (long)blockIdx.x * per + threadIdx.x; i < nvec; i += stride) {
            const uint4 a = __ldg(dy + i);
            const __nv_bfloat16* h = reinterpret_cast<const __nv_bfloat16*>(&a);
            if (relu) {
                const uint4 b = __ldg(y + i);
                const __nv_bfloat16* q = reinterpret_cast<const __nv_bfloat16*>(&b);
                uint4 o;
                __nv_bfloat16* w = reinterpret_cast<__nv_bfloat16*>(&o);
#pragma unroll
                for (int e = 0; e < 8; ++e) {
                    const float v = __bfloat162float(h[e]) * (__bfloat162float(q[e]) > 0.f ? 1.f : 0.f);
                    s[e] += v;
                    w[e] = __float2bfloat16_rn(v);
                }
                g[i] = o;
            } else {
#pragma unroll
                for (int e = 0; e < 8; ++e) s[e] += __bfloat162float(h[e]);
            }
        }
    }
#pragma unroll
    for (int e = 0; e < 8; ++e) rg_sums[threadIdx.x * 8 + e] = s[e];
    __syncthreads();
    for (int c = threadIdx.x; c < groups * 8; c += blockDim.x) {
        float t = 0.f;
        for (int k = c / 8; k < per; k += groups) t += rg_sums[k * 8 + c % 8];
        partial[(size_t)blockIdx.x * groups * 8 + c] = t;
    }
}

// db[c] = sum over blocks of partial[b][c]: one block per channel, a fixed tree
__global__ void __launch_bounds__(128) bias_grad_kernel(const float* __restrict__ partial, float* __restrict__ db, int blocks) {
    __shared__ float red[4];
    const int C = gridDim.x, c = blockIdx.x;
    float t = 0.f;
    for (int b = threadIdx.x; b < blocks; b += 128) t += partial[(size_t)b * C + c];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) t += __shfl_down_sync(0xffffffffu, t, o);
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = t;
    __syncthreads();
    if (threadIdx.x == 0) db[c] = (red[0] + red[1]) + (red[2] + red[3]);
}

}  // namespace

bool conv_wgrad_supported(long Cin, long Cout) {
    return Cin % kCI == 0 && Cout % 16 == 0 && (Cin / kCI) * (Cout / 16) <= 65535;   // one block row per channel tile
}

// Slices: whole rounds of the 296 resident blocks, at most 256 tiles (2^16 voxels) summed in one
// accumulator.  They live in the caller's im2col scratch (27 Cin D H W BF16 elements), which
// holds them (*fits) for all but the smallest volumes; those allocate.
static long wgrad_splits(long D, long H, long W, long Cin, long Cout, bool* fits) {
    const long ntiles = ((W + kTX - 1) / kTX) * ((H + kTY - 1) / kTY) * ((D + kTZ - 1) / kTZ);
    const long chan = Cin / kCI * (Cout / (Cout % 32 == 0 ? 32 : 16)), per = Cout * 27 * Cin;
    const long round = std::max(1L, 296 / chan);
    long splits = round * std::max(1L, (ntiles / round + 255) / 256);
    const long room = 27 * Cin * D * H * W / 2 / per;
    splits = std::max(1L, std::min(splits, ntiles));
    *fits = room >= 1;
    return *fits ? std::min(splits, room) : splits;
}

long conv_wgrad_work(long D, long H, long W, long Cin, long Cout) {
    bool fits;
    const long splits = wgrad_splits(D, H, W, Cin, Cout, &fits);
    return fits ? splits * Cout * 27 * Cin : 0;
}

int launch_conv_wgrad(const __nv_bfloat16* x, const __nv_bfloat16* dy, float* dw, long D, long H, long W, long Cin,
                      long Cout, float* work, cudaStream_t st) {
    WgArgs a{};
    a.x = x;
    a.dy = dy;
    a.D = (int)D; a.H = (int)H; a.W = (int)W; a.Cin = (int)Cin; a.Cout = (int)Cout;
    a.tx = (int)((W + kTX - 1) / kTX);
    a.ty = (int)((H + kTY - 1) / kTY);
    a.ntiles = (long)a.tx * a.ty * ((D + kTZ - 1) / kTZ);
    a.nci = (int)(Cin / kCI);
    const int CO = Cout % 32 == 0 ? 32 : 16;
    const long chan = a.nci * (Cout / CO), per = Cout * 27 * Cin;
    bool fits;
    const long splits = wgrad_splits(D, H, W, Cin, Cout, &fits);
    a.splits = (int)splits;
    float* own = nullptr;
    if (!fits) TIGRE_CUDA(cudaMallocAsync(&own, sizeof(float) * (size_t)(splits * per), st));
    float* ws = own ? own : work;
    a.ws = ws;
    const dim3 grid((unsigned)splits, (unsigned)chan);
    const int smem = 2 * stage_bytes(CO);
    if (CO == 32) {
        TIGRE_CUDA(cudaFuncSetAttribute(conv_wgrad_kernel<32>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
        conv_wgrad_kernel<32><<<grid, kWgThreads, smem, st>>>(a);
    } else {
        TIGRE_CUDA(cudaFuncSetAttribute(conv_wgrad_kernel<16>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
        conv_wgrad_kernel<16><<<grid, kWgThreads, smem, st>>>(a);
    }
    TIGRE_LAUNCHED();
    wgrad_reduce_kernel<<<(unsigned)((per + 255) / 256), 256, 0, st>>>(ws, dw, per, a.splits);
    TIGRE_LAUNCHED();
    if (own) TIGRE_CUDA(cudaFreeAsync(own, st));
    return TIGRE_SUCCESS;
}

}  // namespace tigre

using namespace tigre;

namespace {
long relu_grad_blocks(long n, long C) {
    const int groups = (int)(C / 8), per = 256 / groups * groups;
    return std::max(1L, std::min((n * groups + per - 1) / per, 148L * 4));
}
}  // namespace

extern "C" {

long long tigre_conv3d_relu_grad_work(long n, long C) {
    return n > 0 && C > 0 && C % 8 == 0 && C <= 2048 ? relu_grad_blocks(n, C) * C : 0;
}

int tigre_conv3d_relu_grad(const void* d_dy, const void* d_y, void* d_g, float* d_db, long n, long C, int relu,
                           float* d_work, void* stream) {
    TIGRE_NVTX("tigre_conv3d_relu_grad");
    if (!d_dy || !d_db || !d_work || n <= 0 || C <= 0 || (relu && (!d_y || !d_g)))
        return fail(TIGRE_ERR_BAD_ASSERT, "bad relu_grad arguments");
    if (C % 8 || C > 2048) return fail(TIGRE_ERR_BAD_ASSERT, "relu_grad: channels must be a multiple of 8, at most 2048");
    if (((uintptr_t)d_dy | (uintptr_t)d_y | (uintptr_t)d_g) & 15)
        return fail(TIGRE_ERR_BAD_ASSERT, "relu_grad: buffers must be 16-byte aligned");
    cudaStream_t st = (cudaStream_t)stream;
    const int groups = (int)(C / 8);
    const long blocks = relu_grad_blocks(n, C);
    relu_grad_kernel<<<(unsigned)blocks, 256, 256 * 8 * sizeof(float), st>>>(
        (const uint4*)d_dy, (const uint4*)d_y, (uint4*)d_g, d_work, n * groups, groups, relu ? 1 : 0);
    TIGRE_LAUNCHED();
    bias_grad_kernel<<<(unsigned)C, 128, 0, st>>>(d_work, d_db, (int)blocks);
    TIGRE_LAUNCHED();
    return TIGRE_SUCCESS;
}

}  // extern "C"
