// The glue of the warm-start U-Net's inference pass, fused so that each step is one pass over
// HBM (channels-last BF16 activations, FP32 arithmetic):
//   tigre_unet_pool2      2x2x2 average pooling                  (read 8 voxels, write 1)
//   tigre_unet_up2        nearest 2x upsampling of the deeper level, which the decoder's convolution
//                         reads beside the skip connection       (read 1 voxel, write 8)
//   tigre_unet_up_concat  the same concatenated with the skip connection along channels, where the
//                         convolution does not take two inputs   (one write of the decoder input)
//   tigre_unet_conv_in    the first 3x3x3 convolution (one input channel, FP32 volume rounded to
//                         BF16 on the fly, FP32 accumulation, bias, ReLU)
//   tigre_unet_conv_out   the last 3x3x3 convolution (one output channel) rounded to BF16 as the
//                         convolution output is, plus the residual input volume, FP32 out
// The network's other convolutions are the tensor-core kernels of conv3d*.cu.

#include <cuda_bf16.h>

#include <algorithm>
#include <climits>

#include "tigre_internal.h"

namespace tigre {
namespace {

int grid_for(long n) { return (int)std::min<long>((n + 255) / 256, 148L * 32); }

__device__ __forceinline__ void bf8_to_f(const uint4 v, float (&f)[8]) {
    const uint32_t w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        f[2 * i] = __uint_as_float(w[i] << 16);
        f[2 * i + 1] = __uint_as_float(w[i] & 0xffff0000u);
    }
}

__device__ __forceinline__ uint4 f_to_bf8(const float (&f)[8]) {
    uint32_t w[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const __nv_bfloat162 h = __floats2bfloat162_rn(f[2 * i], f[2 * i + 1]);
        w[i] = *reinterpret_cast<const uint32_t*>(&h);
    }
    return make_uint4(w[0], w[1], w[2], w[3]);
}

// y[z][y][x][c] = mean of x over the 2x2x2 block; one thread per (voxel, 8 channels)
__global__ void pool2_kernel(const uint4* __restrict__ x, uint4* __restrict__ y, int D, int H, int W, int C8) {
    const int d = D / 2, h = H / 2, w = W / 2;
    const long total = (long)d * h * w * C8;
    for (long e = blockIdx.x * (long)blockDim.x + threadIdx.x; e < total; e += (long)gridDim.x * blockDim.x) {
        const int c = (int)(e % C8);
        long v = e / C8;
        const int ox = (int)(v % w), oy = (int)((v / w) % h), oz = (int)(v / ((long)w * h));
        float s[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
#pragma unroll
        for (int k = 0; k < 8; ++k) {
            const int iz = 2 * oz + (k >> 2), iy = 2 * oy + ((k >> 1) & 1), ix = 2 * ox + (k & 1);
            float f[8];
            bf8_to_f(__ldg(x + (((long)iz * H + iy) * W + ix) * C8 + c), f);
#pragma unroll
            for (int j = 0; j < 8; ++j) s[j] += f[j];
        }
#pragma unroll
        for (int j = 0; j < 8; ++j) s[j] *= 0.125f;
        y[e] = f_to_bf8(s);
    }
}

// out[z][y][x][0:Ca] = low[z/2][y/2][x/2][:], out[z][y][x][Ca:Ca+Cb] = skip[z][y][x][:]
__global__ void up_concat_kernel(const uint4* __restrict__ low, int Ca8, const uint4* __restrict__ skip, int Cb8,
                                 uint4* __restrict__ out, int D, int H, int W) {
    const int C8 = Ca8 + Cb8;
    const long total = (long)D * H * W * C8;
    for (long e = blockIdx.x * (long)blockDim.x + threadIdx.x; e < total; e += (long)gridDim.x * blockDim.x) {
        const int c = (int)(e % C8);
        const long v = e / C8;
        uint4 val;
        if (c < Ca8) {
            const int x = (int)(v % W), y = (int)((v / W) % H), z = (int)(v / ((long)W * H));
            val = __ldg(low + ((((long)(z >> 1) * (H >> 1) + (y >> 1)) * (W >> 1) + (x >> 1)) * Ca8 + c));
        } else {
            val = __ldg(skip + v * Cb8 + (c - Ca8));
        }
        out[e] = val;
    }
}

// out[z][y][x] = low[z/2][y/2][x/2]: one thread per 16 bytes of low, eight stores
__global__ void __launch_bounds__(256) up2_kernel(const uint4* __restrict__ low, uint4* __restrict__ out, int d, int h, int w,
                                                  int C8) {
    const long row = (long)w * C8, total = (long)d * h * row;
    for (long e = blockIdx.x * (long)blockDim.x + threadIdx.x; e < total; e += (long)gridDim.x * blockDim.x) {
        const long v = e / C8;
        const int c = (int)(e - v * C8), x = (int)(v % w);
        const long zy = v / w;
        const int y = (int)(zy % h), z = (int)(zy / h);
        const uint4 val = __ldg(low + e);
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            uint4* o = out + (((2L * z + (k >> 1)) * (2 * h) + 2 * y + (k & 1)) * (2L * w) + 2 * x) * C8 + c;
            o[0] = val;
            o[C8] = val;
        }
    }
}

// First convolution: one input channel (vol, FP32, rounded to BF16), COUT outputs.  The sum of an
// output starts from its bias and takes the 27 taps in order, each by one FP32 fused multiply-add:
// what the network computes behind it depends on every rounding here (the BF16 steps of 14 layers), so
// the order is part of the result, and the tensor cores, which sum in one of their own, are not used.
// A block marches a 32 x 16 tile of (x, y) down a chunk of slices, three staged at a time and the next one
// on its way in registers; a thread owns four rows of one x and 16 channels, so that a tap's weights (one
// broadcast 16-byte load per four) serve four voxels and a voxel up to nine taps, two channels to an
// instruction.  Bound by the FP32 pipe, 27 COUT multiply-adds a voxel: 256^3, 16 channels 322 us, 201 at its
// full rate (one voxel a thread with 27 bounds-tested loads 785; on the tensor cores, in their order, 203);
// 64^3 11 us (19).  Four blocks per SM 374 (spills); two rows a thread at 5 or 6 blocks 341 / 367.
constexpr int kInX = 32, kInY = 16, kInRows = 4, kInBlocks = 3;
constexpr int kInThreads = kInX * kInY / kInRows;
constexpr int kInHalo = (kInX + 2) * (kInY + 2), kInFetch = (kInHalo + kInThreads - 1) / kInThreads;

template <int COUT>
__global__ void __launch_bounds__(kInThreads, kInBlocks) conv_in_kernel(const float* __restrict__ vol,
                                                                const __nv_bfloat16* __restrict__ w,
                                                                const float* __restrict__ b, __nv_bfloat16* __restrict__ y,
                                                                int D, int H, int W, int tx, int ty, int zc, int relu) {
    constexpr int CG = COUT < 16 ? COUT : 16;   // channels of a thread at a time
    __shared__ float ring[3][kInHalo];
    __shared__ __align__(16) float sw[27][COUT];
    __shared__ float sb[COUT];
    const int tid = threadIdx.x, lx = tid % kInX, ly = tid / kInX * kInRows;
    const int bx = (int)(blockIdx.x % (unsigned)tx), bt = (int)(blockIdx.x / (unsigned)tx);
    const int x0 = bx * kInX, y0 = bt % ty * kInY, z0 = bt / ty * zc, zend = min(z0 + zc, D);
    for (int i = tid; i < 27 * COUT; i += kInThreads) sw[i % 27][i / 27] = __bfloat162float(w[i]);
    for (int i = tid; i < COUT; i += kInThreads) sb[i] = b ? b[i] : 0.f;
    float next[kInFetch];
    auto fetch = [&](int z) {
#pragma unroll
        for (int k = 0; k < kInFetch; ++k) {
            const int e = tid + k * kInThreads, gy = y0 + e / (kInX + 2) - 1, gx = x0 + e % (kInX + 2) - 1;
            const bool ok = e < kInHalo && z >= 0 && z < D && gy >= 0 && gy < H && gx >= 0 && gx < W;
            next[k] = ok ? __ldg(vol + ((long)z * H + gy) * W + gx) : 0.f;
        }
    };
    auto put = [&](int z) {
#pragma unroll
        for (int k = 0; k < kInFetch; ++k) {
            const int e = tid + k * kInThreads;
            if (e < kInHalo) ring[(z + 3) % 3][e] = __bfloat162float(__float2bfloat16(next[k]));
        }
    };
    fetch(z0 - 1);
    put(z0 - 1);
    fetch(z0);
    put(z0);
    fetch(z0 + 1);
    for (int z = z0; z < zend; ++z) {
        put(z + 1);
        __syncthreads();
        fetch(z + 2);
        const int gx = x0 + lx;
#pragma unroll 1
        for (int cg = 0; cg < COUT; cg += CG) {
            float2 acc[kInRows][CG / 2];
#pragma unroll
            for (int r = 0; r < kInRows; ++r)
#pragma unroll
                for (int c = 0; c < CG / 2; ++c) acc[r][c] = make_float2(sb[cg + 2 * c], sb[cg + 2 * c + 1]);
#pragma unroll 1
            for (int dz = 0; dz < 3; ++dz) {
                const float* in = &ring[(z + dz + 2) % 3][ly * (kInX + 2) + lx];
                float v[kInRows + 2][3];
#pragma unroll
                for (int r = 0; r < kInRows + 2; ++r)
#pragma unroll
                    for (int dx = 0; dx < 3; ++dx) v[r][dx] = in[r * (kInX + 2) + dx];
#pragma unroll
                for (int t = 0; t < 9; ++t) {
                    const float4* wt = reinterpret_cast<const float4*>(&sw[9 * dz + t][cg]);
#pragma unroll
                    for (int c = 0; c < CG / 4; ++c) {
                        const float4 q = wt[c];
#pragma unroll
                        for (int r = 0; r < kInRows; ++r) {
                            const float2 in2 = make_float2(v[r + t / 3][t % 3], v[r + t / 3][t % 3]);
                            acc[r][2 * c] = __ffma2_rn(make_float2(q.x, q.y), in2, acc[r][2 * c]);
                            acc[r][2 * c + 1] = __ffma2_rn(make_float2(q.z, q.w), in2, acc[r][2 * c + 1]);
                        }
                    }
                }
            }
#pragma unroll
            for (int r = 0; r < kInRows; ++r) {
                const int gy = y0 + ly + r;
                if (gx >= W || gy >= H) continue;
                uint4* o = reinterpret_cast<uint4*>(y + (((long)z * H + gy) * W + gx) * COUT + cg);
#pragma unroll
                for (int c = 0; c < CG / 8; ++c) {
                    float f[8];
#pragma unroll
                    for (int j = 0; j < 4; ++j) {
                        const float2 a = acc[r][4 * c + j];
                        f[2 * j] = relu ? fmaxf(a.x, 0.f) : a.x;
                        f[2 * j + 1] = relu ? fmaxf(a.y, 0.f) : a.y;
                    }
                    o[c] = f_to_bf8(f);
                }
            }
        }
        __syncthreads();   // slice z - 1 is replaced by z + 2
    }
}

// Last convolution: CIN input channels -> 1, rounded to BF16, plus the residual volume (FP32).  The sum
// starts from the bias and takes the taps in order and a tap's channels in order, by FP32 fused
// multiply-adds (as the first convolution, for the same reason).  A block marches a 32 x 16 tile of (x, y)
// down a chunk of slices, one input slice staged and the next on its way; a slice's 9 CIN products go
// to three output slices at once, whose sums a thread carries for four neighbouring x: the weights of the
// three dz are one broadcast 16-byte load for 12 multiply-adds, and a staged voxel is read three times instead of 27.
// The staged voxels are kept in planes of eight channels, every fourth x together, which makes the
// 16-byte loads of eight threads one 128-byte run.  Bound by instruction issue, 27 CIN multiply-adds and
// 9 CIN conversions an output voxel: 256^3, 16 channels 494 us (one voxel a thread 1362; on the tensor cores 336),
// 64^3 29 us (31).  3 / 5 blocks per SM 530 / 515; two voxels to an instruction, which doubles the weights'
// loads, 510 to 569.
constexpr int kOutX = 32, kOutY = 16, kOutV = 4, kOutThreads = kOutX * kOutY / kOutV;
constexpr int out_blocks(int cin) { return cin <= 16 ? 4 : 2; }       // resident blocks per SM
constexpr int kOutRow = kOutV * (kOutX / kOutV + 1);                  // 16-byte places of a staged row
constexpr int out_plane() { return (kOutY + 2) * kOutRow; }           // ... of a plane
constexpr size_t out_smem(int cin) { return 16 * (size_t)(2 * cin / 8 * out_plane() + 9 * cin); }

template <int CIN>
__global__ void __launch_bounds__(kOutThreads, out_blocks(CIN)) conv_out_kernel(const __nv_bfloat16* __restrict__ x,
                                                                                  const __nv_bfloat16* __restrict__ w, float b,
                                                                                  const float* __restrict__ vol,
                                                                                  float* __restrict__ out, int D, int H, int W,
                                                                                  int tx, int ty, int zc) {
    constexpr int NG = CIN / 8, PL = out_plane();
    extern __shared__ __align__(16) uint4 out_sm[];   // two slices of NG planes, then the weights
    float4* sw = reinterpret_cast<float4*>(out_sm + 2 * NG * PL);   // [dy, dx][c]: dz = 0, 1, 2
    const int tid = threadIdx.x, xg = tid % (kOutX / kOutV), row = tid / (kOutX / kOutV);
    const int bx = (int)(blockIdx.x % (unsigned)tx), bt = (int)(blockIdx.x / (unsigned)tx);
    const int x0 = bx * kOutX, y0 = bt % ty * kOutY, z0 = bt / ty * zc, zend = min(z0 + zc, D);
    for (int i = tid; i < 9 * CIN; i += kOutThreads)
        sw[i] = make_float4(__bfloat162float(w[i]), __bfloat162float(w[9 * CIN + i]), __bfloat162float(w[18 * CIN + i]), 0.f);
    auto stage = [&](int s) {
        const uint32_t base = (uint32_t)__cvta_generic_to_shared(out_sm + (s & 1) * NG * PL);
        for (int e = tid; e < (kOutY + 2) * (kOutX + 2) * NG; e += kOutThreads) {
            const int g = e % NG, v = e / NG, px = v % (kOutX + 2), r = v / (kOutX + 2);
            const int gx = x0 + px - 1, gy = y0 + r - 1;
            const bool ok = gx >= 0 && gx < W && gy >= 0 && gy < H;
            const __nv_bfloat16* src = ok ? x + (((long)s * H + gy) * W + gx) * CIN + 8 * g : x;
            const int at = g * PL + r * kOutRow + px % kOutV * (kOutX / kOutV + 1) + px / kOutV;
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(base + 16u * (uint32_t)at), "l"(src),
                         "r"(ok ? 16 : 0)
                         : "memory");
        }
        asm volatile("cp.async.commit_group;\n" ::: "memory");
    };
    // sums of the output slices s - 1, s and s + 1 (s: input slice)
    float a0[kOutV], a1[kOutV], a2[kOutV];
#pragma unroll
    for (int k = 0; k < kOutV; ++k) a0[k] = a1[k] = b;
    const int first = max(z0 - 1, 0), last = min(zend, D - 1);
    stage(first);
    for (int s = first; s <= last; ++s) {
        if (s < last) {
            stage(s + 1);
            asm volatile("cp.async.wait_group 1;\n" ::: "memory");
        } else {
            asm volatile("cp.async.wait_group 0;\n" ::: "memory");
        }
        __syncthreads();
        const uint4* in = out_sm + (s & 1) * NG * PL + row * kOutRow + xg;
#pragma unroll
        for (int k = 0; k < kOutV; ++k) a2[k] = b;
#pragma unroll 1
        for (int dy = 0; dy < 3; ++dy) {
            uint4 v[kOutV + 2][NG];
#pragma unroll
            for (int k = 0; k < kOutV + 2; ++k)
#pragma unroll
                for (int g = 0; g < NG; ++g)
                    v[k][g] = in[g * PL + dy * kOutRow + k % kOutV * (kOutX / kOutV + 1) + k / kOutV];
#pragma unroll
            for (int dx = 0; dx < 3; ++dx)
#pragma unroll
                for (int c = 0; c < CIN; ++c) {
                    const float4 q = sw[(3 * dy + dx) * CIN + c];
#pragma unroll
                    for (int k = 0; k < kOutV; ++k) {
                        const uint4& u = v[k + dx][c / 8];
                        const uint32_t h = c % 8 < 2 ? u.x : c % 8 < 4 ? u.y : c % 8 < 6 ? u.z : u.w;
                        const float f = __uint_as_float(c % 2 ? h & 0xffff0000u : h << 16);
                        a2[k] = fmaf(q.x, f, a2[k]);
                        a1[k] = fmaf(q.y, f, a1[k]);
                        a0[k] = fmaf(q.z, f, a0[k]);
                    }
                }
        }
        const int gy = y0 + row;
#pragma unroll
        for (int k = 0; k < kOutV; ++k) {
            const int gx = x0 + kOutV * xg + k;
            auto emit = [&](int z, float acc) {
                const long i = ((long)z * H + gy) * W + gx;
                out[i] = vol[i] + __bfloat162float(__float2bfloat16(acc));
            };
            if (gx < W && gy < H) {
                if (s - 1 >= z0) emit(s - 1, a0[k]);
                if (s == D - 1 && s < zend) emit(s, a1[k]);   // no slice above the last
            }
            a0[k] = a1[k];
            a1[k] = a2[k];
        }
        __syncthreads();   // slice s is replaced by s + 2
    }
}

// Slices per block of a march: the fewest steps over the rounds of resident blocks, where a chunk of zc
// slices takes zc + extra steps (64^3, last convolution: chunks of 32 slices 95 us, of this rule 29).
int march_chunk(long tiles, long D, long resident, int extra) {
    int best = 1;
    double least = 0.0;
    for (int zc = 1; zc <= 64; zc += zc < 16 ? 1 : zc / 8) {
        const long blocks = tiles * ((D + zc - 1) / zc);
        const double cost = (double)((blocks + 148 * resident - 1) / (148 * resident)) * (zc + extra);
        if (zc == 1 || cost < least) { least = cost; best = zc; }
    }
    return best;
}

bool aligned16(const void* p) { return ((uintptr_t)p & 15) == 0; }

}  // namespace
}  // namespace tigre

using namespace tigre;

extern "C" {

int tigre_unet_pool2(const void* d_x, void* d_y, long D, long H, long W, long C, void* stream) {
    if (!d_x || !d_y || D <= 0 || H <= 0 || W <= 0 || D % 2 || H % 2 || W % 2 || C <= 0 || C % 8 ||
        !aligned16(d_x) || !aligned16(d_y))
        return fail(TIGRE_ERR_BAD_ASSERT, "unet pool2: even sizes, C % 8 == 0 and 16-byte aligned buffers");
    const long n = (D / 2) * (H / 2) * (W / 2) * (C / 8);
    pool2_kernel<<<grid_for(n), 256, 0, (cudaStream_t)stream>>>((const uint4*)d_x, (uint4*)d_y, (int)D, (int)H, (int)W,
                                                              (int)(C / 8));
    TIGRE_LAUNCHED();
    return TIGRE_SUCCESS;
}

int tigre_unet_up_concat(const void* d_low, long Ca, const void* d_skip, long Cb, void* d_out, long D, long H, long W,
                         void* stream) {
    if (!d_low || !d_skip || !d_out || D % 2 || H % 2 || W % 2 || D <= 0 || H <= 0 || W <= 0 || Ca % 8 || Cb % 8 ||
        Ca <= 0 || Cb <= 0 || !aligned16(d_low) || !aligned16(d_skip) || !aligned16(d_out))
        return fail(TIGRE_ERR_BAD_ASSERT, "unet up_concat: even sizes, channels % 8 == 0, 16-byte aligned buffers");
    const long n = D * H * W * ((Ca + Cb) / 8);
    up_concat_kernel<<<grid_for(n), 256, 0, (cudaStream_t)stream>>>((const uint4*)d_low, (int)(Ca / 8),
                                                                  (const uint4*)d_skip, (int)(Cb / 8), (uint4*)d_out,
                                                                  (int)D, (int)H, (int)W);
    TIGRE_LAUNCHED();
    return TIGRE_SUCCESS;
}

int tigre_unet_up2(const void* d_low, void* d_out, long D, long H, long W, long C, void* stream) {
    if (!d_low || !d_out || D % 2 || H % 2 || W % 2 || D <= 0 || H <= 0 || W <= 0 || C % 8 || C <= 0 || !aligned16(d_low) ||
        !aligned16(d_out))
        return fail(TIGRE_ERR_BAD_ASSERT, "unet up2: even sizes, channels % 8 == 0, 16-byte aligned buffers");
    const long n = (D / 2) * (H / 2) * (W / 2) * (C / 8);
    up2_kernel<<<grid_for(n), 256, 0, (cudaStream_t)stream>>>((const uint4*)d_low, (uint4*)d_out, (int)(D / 2), (int)(H / 2),
                                                            (int)(W / 2), (int)(C / 8));
    TIGRE_LAUNCHED();
    return TIGRE_SUCCESS;
}

int tigre_unet_conv_in(const float* d_vol, const void* d_w, const float* d_b, void* d_y, long D, long H, long W,
                       long Cout, int relu, void* stream) {
    if (!d_vol || !d_w || !d_y || D <= 0 || H <= 0 || W <= 0 || !aligned16(d_y))
        return fail(TIGRE_ERR_BAD_ASSERT, "unet conv_in: bad arguments");
    cudaStream_t st = (cudaStream_t)stream;
    const __nv_bfloat16* w = (const __nv_bfloat16*)d_w;
    __nv_bfloat16* y = (__nv_bfloat16*)d_y;
    const long tx = (W + kInX - 1) / kInX, ty = (H + kInY - 1) / kInY;
    const int zc = march_chunk(tx * ty, D, kInBlocks, 1);
    const long blocks = tx * ty * ((D + zc - 1) / zc);
    if (blocks > INT_MAX || D > INT_MAX - 64 || H > INT_MAX - 64 || W > INT_MAX - 128)
        return fail(TIGRE_ERR_BAD_ASSERT, "unet conv_in: volume too large");
    auto go = [&](auto kern) { kern<<<(unsigned)blocks, kInThreads, 0, st>>>(d_vol, w, d_b, y, (int)D, (int)H, (int)W, (int)tx, (int)ty, zc, relu); };
    if (Cout == 8) go(conv_in_kernel<8>);
    else if (Cout == 16) go(conv_in_kernel<16>);
    else if (Cout == 32) go(conv_in_kernel<32>);
    else return fail(TIGRE_ERR_BAD_ASSERT, "unet conv_in: Cout must be 8, 16 or 32");
    TIGRE_LAUNCHED();
    return TIGRE_SUCCESS;
}

int tigre_unet_conv_out(const void* d_x, long Cin, const void* d_w, float b, const float* d_vol, float* d_out, long D,
                        long H, long W, void* stream) {
    if (!d_x || !d_w || !d_vol || !d_out || D <= 0 || H <= 0 || W <= 0 || !aligned16(d_x))
        return fail(TIGRE_ERR_BAD_ASSERT, "unet conv_out: bad arguments");
    cudaStream_t st = (cudaStream_t)stream;
    const __nv_bfloat16* x = (const __nv_bfloat16*)d_x;
    const __nv_bfloat16* w = (const __nv_bfloat16*)d_w;
    const long tx = (W + kOutX - 1) / kOutX, ty = (H + kOutY - 1) / kOutY;
    const int zc = march_chunk(tx * ty, D, out_blocks((int)Cin), 2);
    const long blocks = tx * ty * ((D + zc - 1) / zc);
    if (blocks > INT_MAX || D > INT_MAX - 64 || H > INT_MAX - 64 || W > INT_MAX - 128)
        return fail(TIGRE_ERR_BAD_ASSERT, "unet conv_out: volume too large");
    auto go = [&](auto kern) -> int {
        const int smem = (int)out_smem((int)Cin);
        TIGRE_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
        kern<<<(unsigned)blocks, kOutThreads, smem, st>>>(x, w, b, d_vol, d_out, (int)D, (int)H, (int)W, (int)tx, (int)ty, zc);
        TIGRE_LAUNCHED();
        return TIGRE_SUCCESS;
    };
    if (Cin == 8) return go(conv_out_kernel<8>);
    if (Cin == 16) return go(conv_out_kernel<16>);
    if (Cin == 32) return go(conv_out_kernel<32>);
    return fail(TIGRE_ERR_BAD_ASSERT, "unet conv_out: Cin must be 8, 16 or 32");
}

}  // extern "C"
