// The glue of the warm-start U-Net's inference pass, fused so that each step is one pass over
// HBM (channels-last BF16 activations, FP32 arithmetic):
//   tigre_unet_pool2      2x2x2 average pooling                  (read 8 voxels, write 1)
//   tigre_unet_up_concat  nearest 2x upsampling of the deeper level concatenated with the skip
//                         connection along channels              (one write of the decoder input)
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

__device__ __forceinline__ void mma_bf16(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0,
                                         uint32_t b1) {
    asm volatile(
        "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
        : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
        : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

__device__ __forceinline__ uint32_t pack_bf16(__nv_bfloat16 lo, __nv_bfloat16 hi) {
    return (uint32_t)__bfloat16_as_ushort(lo) | ((uint32_t)__bfloat16_as_ushort(hi) << 16);
}

// First convolution: one input channel (vol, FP32, rounded to BF16), COUT outputs, as warp-level
// m16n8k16 products of 16 voxels along x with the taps as K.  Per (dz, dy) row the three dx taps
// take two K pairs, (x-1, x) and (x+1, -), so that an operand register is one 32-bit word of the
// staged row; the row is kept twice, the second copy shifted by one voxel, which makes the pair of
// any x an aligned word.  18 of 24 K pairs carry weights; the others and the unused halves are
// zeroed on both sides.  A block marches a 64 x 8 tile of (x, y) down kInZ slices, three staged at a
// time; output column c of tile t is channel 2 NT (c / 2) + 2 t + c % 2, so a thread stores
// 4 NT contiguous bytes.
// 256^3, 16 channels: 205 us, 604 MB written and read at 2.9 TB/s (scalar FMAs, 27 bounds-tested loads a
// voxel: 806 us); bound by the shared-memory loads of the operands and the staging.
constexpr int kInX = 64, kInY = 8, kInZ = 16;
constexpr int kInWords = kInX / 2 + 2;                 // words of one staged row and copy
constexpr int kInPitch = 2 * kInWords + 1;             // both copies (odd: rows fall in other banks)

template <int COUT>
__global__ void __launch_bounds__(256) conv_in_kernel(const float* __restrict__ vol, const __nv_bfloat16* __restrict__ w,
                                                      const float* __restrict__ b, __nv_bfloat16* __restrict__ y,
                                                      int D, int H, int W, int tx, int ty, int relu) {
    constexpr int NT = COUT / 8;
    __shared__ uint32_t ring[3][kInY + 2][kInPitch];
    const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5, g = lane >> 2, q = lane & 3;
    const int bx = (int)(blockIdx.x % (unsigned)tx), bt = (int)(blockIdx.x / (unsigned)tx);
    const int x0 = bx * kInX, y0 = bt % ty * kInY, z0 = bt / ty * kInZ, zend = min(z0 + kInZ, D);
    auto channel = [](int t, int c) { return 2 * NT * (c >> 1) + 2 * t + (c & 1); };
    // weights: K pair slot s = 8 kstep + 4 half + q holds taps (2 (s % 2), 2 (s % 2) + 1) of row s / 2
    uint32_t wb[3][2][NT];
    float bias[NT][2];
#pragma unroll
    for (int t = 0; t < NT; ++t) {
#pragma unroll
        for (int k = 0; k < 3; ++k)
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const int s = 8 * k + 4 * h + q, row = s >> 1;
                const __nv_bfloat16* src = w + channel(t, g) * 27 + row * 3;
                const __nv_bfloat16 zero = __float2bfloat16(0.f);
                wb[k][h][t] = row >= 9 ? 0u : (s & 1) ? pack_bf16(src[2], zero) : pack_bf16(src[0], src[1]);
            }
#pragma unroll
        for (int e = 0; e < 2; ++e) bias[t][e] = b ? b[channel(t, 2 * q + e)] : 0.f;
    }
    // stages slice z: word j of copy 0 = (v[2j], v[2j+1]), of copy 1 = (v[2j+1], v[2j+2]), v[0] at x0 - 1
    auto stage = [&](int z) {
        const bool zin = z >= 0 && z < D;
        uint32_t(*dst)[kInPitch] = ring[(z + 3) % 3];
        for (int e = tid; e < (kInY + 2) * kInWords; e += 256) {
            const int r = e / kInWords, j = e - r * kInWords, gy = y0 + r - 1;
            __nv_bfloat16 v[3];
#pragma unroll
            for (int k = 0; k < 3; ++k) {
                const int gx = x0 - 1 + 2 * j + k;
                const bool ok = zin && gy >= 0 && gy < H && gx >= 0 && gx < W;
                v[k] = __float2bfloat16(ok ? __ldg(vol + ((long)z * H + gy) * W + gx) : 0.f);
            }
            dst[r][j] = pack_bf16(v[0], v[1]);
            dst[r][kInWords + j] = pack_bf16(v[1], v[2]);
        }
    };
    stage(z0 - 1);
    stage(z0);
    for (int z = z0; z < zend; ++z) {
        stage(z + 1);
        __syncthreads();
        const int gy = y0 + wid;
        if (gy < H) {
            const uint32_t* rows[3][2];   // this thread's K pair slots
            uint32_t mask[3][2];
#pragma unroll
            for (int k = 0; k < 3; ++k)
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    const int s = 8 * k + 4 * h + q, row = min(s >> 1, 8);
                    rows[k][h] = &ring[(z + row / 3 + 2) % 3][wid + row % 3][(s & 1) + (g & 1) * kInWords + (g >> 1)];
                    mask[k][h] = s >= 18 ? 0u : (s & 1) ? 0xffffu : 0xffffffffu;
                }
            __nv_bfloat16* o = y + (((long)z * H + gy) * W + x0) * COUT;
#pragma unroll
            for (int m = 0; m < kInX / 16; ++m) {
                if (x0 + 16 * m >= W) break;
                float c[NT][4];
#pragma unroll
                for (int t = 0; t < NT; ++t) {
                    c[t][0] = c[t][2] = bias[t][0];
                    c[t][1] = c[t][3] = bias[t][1];
                }
#pragma unroll
                for (int k = 0; k < 3; ++k) {
                    const uint32_t a0 = rows[k][0][8 * m] & mask[k][0], a1 = rows[k][0][8 * m + 4] & mask[k][0];
                    const uint32_t a2 = rows[k][1][8 * m] & mask[k][1], a3 = rows[k][1][8 * m + 4] & mask[k][1];
#pragma unroll
                    for (int t = 0; t < NT; ++t) mma_bf16(c[t], a0, a1, a2, a3, wb[k][0][t], wb[k][1][t]);
                }
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    const int x = 16 * m + g + 8 * h;
                    if (x0 + x < W) {
                        uint32_t v[NT];
#pragma unroll
                        for (int t = 0; t < NT; ++t) {
                            const float lo = relu ? fmaxf(c[t][2 * h], 0.f) : c[t][2 * h];
                            const float hi = relu ? fmaxf(c[t][2 * h + 1], 0.f) : c[t][2 * h + 1];
                            const __nv_bfloat162 p = __floats2bfloat162_rn(lo, hi);
                            v[t] = *reinterpret_cast<const uint32_t*>(&p);
                        }
                        uint32_t* dst = reinterpret_cast<uint32_t*>(o + (long)x * COUT) + NT * q;
                        if constexpr (NT == 4) *reinterpret_cast<uint4*>(dst) = make_uint4(v[0], v[1], v[2], v[3]);
                        else if constexpr (NT == 2) *reinterpret_cast<uint2*>(dst) = make_uint2(v[0], v[1]);
                        else dst[0] = v[0];
                    }
                }
            }
        }
        __syncthreads();   // slice z - 1 is replaced by z + 2
    }
}

// Last convolution: CIN input channels -> 1, rounded to BF16, plus the residual volume (FP32).  The
// products run on the warp-level tensor cores with the three rows dy in K and the nine taps (dz, dx) as
// output columns,
//     P[v][dz, dx] = sum_dy sum_c x[v + dy][c] w[dz, dy, dx][c],   out[v] = b + sum P[v + (dz, dx)][dz, dx],
// so that every input voxel's operands are loaded once (1.5 times, with the warps' edge rows), used
// for three rows, and nine words per voxel pass through shared memory instead of 27.  A block marches a
// 62 x 8 tile of (x, y) down kOutZ slices: per input slice, a warp takes 16 x and four of the rows, P goes to
// shared memory as [tap][row][x] (kOutPlane words a tap, which with the pitch leaves the fragments' stores and
// the sums' loads free of bank conflicts), and each thread adds the three dx of each dz into the three
// output slices that the input slice touches.  K index 2 q + e of the low half is channel 4 q + e of a
// 16-channel step, of the high half channel 4 q + 2 + e: a thread's operands are one 8-byte load per voxel.
// 256^3, 16 channels: 336 us (27 tap columns, one row at a time: 498); bound by the latency of the loads, all
// issued before the first product, and of the two barriers a slice.  2 / 4 / 5 blocks per SM 433 / 489 / 552;
// rows loaded one ahead in a window of four at 3 or 4 blocks per SM 455 / 442.
constexpr int kOutX = 62, kOutY = 8, kOutZ = 32, kOutPitch = 66, kOutPlane = kOutY * kOutPitch + 4;

template <int CIN>
__global__ void __launch_bounds__(256, CIN <= 16 ? 3 : 1) conv_out_kernel(const __nv_bfloat16* __restrict__ x,
                                                       const __nv_bfloat16* __restrict__ w, float b,
                                                       const float* __restrict__ vol, float* __restrict__ out, int D,
                                                       int H, int W, int tx, int ty) {
    constexpr int KS = (CIN + 15) / 16;        // K steps (8 channels: one step, its high half zero)
    constexpr int CQ = CIN >= 16 ? 4 : 2;      // channels of a step that a thread holds
    constexpr int RW = kOutY / 2;              // rows of a warp
    __shared__ float P[9 * kOutPlane];         // [tap][kOutY][kOutPitch]
    const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5, g = lane >> 2, q = lane & 3;
    const int bx = (int)(blockIdx.x % (unsigned)tx), bt = (int)(blockIdx.x / (unsigned)tx);
    const int x0 = bx * kOutX, y0 = bt % ty * kOutY, z0 = bt / ty * kOutZ, zend = min(z0 + kOutZ, D);
    uint32_t wb[KS][3][2][2];                  // [step][dy][column tile][K half]
#pragma unroll
    for (int k = 0; k < KS; ++k)
#pragma unroll
        for (int dy = 0; dy < 3; ++dy)
#pragma unroll
            for (int t = 0; t < 2; ++t) {
                const int n = 8 * t + g, tap = n < 9 ? (n / 3 * 3 + dy) * 3 + n % 3 : 0;
                const __nv_bfloat16* src = w + tap * CIN + 16 * k + CQ * q;
                wb[k][dy][t][0] = n < 9 ? pack_bf16(src[0], src[1]) : 0u;
                wb[k][dy][t][1] = n < 9 && CQ == 4 ? pack_bf16(src[CQ - 2], src[CQ - 1]) : 0u;
            }
    // the thread's two output voxels and their sums for slices s - 1, s, s + 1 (s: input slice)
    const int ox = tid & 63, oy = tid >> 6;    // rows oy and oy + 4
    float o0[2] = {0.f, 0.f}, o1[2] = {0.f, 0.f}, o2[2];
    const int xb = (wid & 3) * 16, rb = (wid >> 2) * RW;
    for (int s = max(z0 - 1, 0); s <= min(zend, D - 1); ++s) {
        uint32_t a[RW + 2][KS][2][2];          // [input row rb - 1 + j][step][voxel g / g + 8][K half]
#pragma unroll
        for (int j = 0; j < RW + 2; ++j)
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const int gy = y0 + rb + j - 1, gx = x0 + xb + g + 8 * h - 1;
                const bool ok = gy >= 0 && gy < H && gx >= 0 && gx < W;
                const __nv_bfloat16* src = x + (((long)s * H + (ok ? gy : 0)) * W + (ok ? gx : 0)) * CIN + CQ * q;
#pragma unroll
                for (int k = 0; k < KS; ++k) {
                    if constexpr (CQ == 4) {
                        const uint2 v = ok ? __ldg(reinterpret_cast<const uint2*>(src + 16 * k)) : make_uint2(0u, 0u);
                        a[j][k][h][0] = v.x;
                        a[j][k][h][1] = v.y;
                    } else {
                        a[j][k][h][0] = ok ? __ldg(reinterpret_cast<const uint32_t*>(src)) : 0u;
                        a[j][k][h][1] = 0u;
                    }
                }
            }
#pragma unroll
        for (int r = 0; r < RW; ++r)
#pragma unroll
            for (int t = 0; t < 2; ++t) {
                float c[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
                for (int dy = 0; dy < 3; ++dy)
#pragma unroll
                    for (int k = 0; k < KS; ++k) {
                        const uint32_t(&f)[2][2] = a[r + dy][k];
                        mma_bf16(c, f[0][0], f[1][0], f[0][1], f[1][1], wb[k][dy][t][0], wb[k][dy][t][1]);
                    }
                float* d = P + (8 * t + 2 * q) * kOutPlane + (rb + r) * kOutPitch + xb + g;
                if (t == 0 || q == 0) {        // column 8 is the last
                    d[0] = c[0];
                    d[8] = c[2];
                }
                if (t == 0) {
                    d[kOutPlane] = c[1];
                    d[kOutPlane + 8] = c[3];
                }
            }
        __syncthreads();
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            o2[h] = 0.f;
            if (ox < kOutX) {
                float sum[3] = {0.f, 0.f, 0.f};
#pragma unroll
                for (int t = 0; t < 9; ++t) sum[t / 3] += P[t * kOutPlane + (oy + 4 * h) * kOutPitch + ox + t % 3];
                o0[h] += sum[2];   // dz = 2: input slice s is z + 1 of output slice s - 1
                o1[h] += sum[1];
                o2[h] = sum[0];
                const int gx = x0 + ox, gy = y0 + oy + 4 * h;
                auto put = [&](int z, float acc) {
                    const long i = ((long)z * H + gy) * W + gx;
                    out[i] = __ldg(vol + i) + __bfloat162float(__float2bfloat16(b + acc));
                };
                if (gx < W && gy < H) {
                    if (s - 1 >= z0) put(s - 1, o0[h]);
                    if (s == D - 1 && s < zend) put(s, o1[h]);   // no slice above the last
                }
            }
            o0[h] = o1[h];
            o1[h] = o2[h];
        }
        __syncthreads();   // P is rewritten for the next slice
    }
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
    const long tx = (W + kInX - 1) / kInX, ty = (H + kInY - 1) / kInY, blocks = tx * ty * ((D + kInZ - 1) / kInZ);
    if (blocks > INT_MAX || D > INT_MAX - 64 || H > INT_MAX - 64 || W > INT_MAX - 128)
        return fail(TIGRE_ERR_BAD_ASSERT, "unet conv_in: volume too large");
    auto go = [&](auto kern) { kern<<<(unsigned)blocks, 256, 0, st>>>(d_vol, w, d_b, y, (int)D, (int)H, (int)W, (int)tx, (int)ty, relu); };
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
    const long tx = (W + kOutX - 1) / kOutX, ty = (H + kOutY - 1) / kOutY, blocks = tx * ty * ((D + kOutZ - 1) / kOutZ);
    if (blocks > INT_MAX || D > INT_MAX - 64 || H > INT_MAX - 64 || W > INT_MAX - 128)
        return fail(TIGRE_ERR_BAD_ASSERT, "unet conv_out: volume too large");
    auto go = [&](auto kern) -> int {
        kern<<<(unsigned)blocks, 256, 0, st>>>(x, w, b, d_vol, d_out, (int)D, (int)H, (int)W, (int)tx, (int)ty);
        TIGRE_LAUNCHED();
        return TIGRE_SUCCESS;
    };
    if (Cin == 8) return go(conv_out_kernel<8>);
    if (Cin == 16) return go(conv_out_kernel<16>);
    if (Cin == 32) return go(conv_out_kernel<32>);
    return fail(TIGRE_ERR_BAD_ASSERT, "unet conv_out: Cin must be 8, 16 or 32");
}

}  // extern "C"
