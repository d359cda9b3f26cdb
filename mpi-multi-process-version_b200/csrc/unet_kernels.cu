// Forward and backward kernels of the warm-start surrogate (a 4-level U-Net
// over NHWC bfloat16 images, FP32 accumulation).  No counterpart in the
// reference, which always starts from the conduction state of initial()
// (natural-convection_2dim_mono.f90:199-240).
//
// 3x3 convolutions are implicit GEMMs on the tensor cores (bf16 inputs, FP32
// accumulators), from pixel tiles that serve all nine taps (tcgen05, TMA copies):
//   forward      M = pixels, N = Cout, K = 9 Cin;
//   data grad    the same kernel on dL/dz with the flipped, transposed weights;
//   weight grad  M = Cout, N = 9 Cin, K = pixels, split over pixel tiles into
//                FP32 partials that a second kernel sums in a fixed order
//                (deterministic).
// k_conv3x3 (mma.sync) takes pixels in a row, across images, for many images far
// smaller than a tile.
// Elementwise work (SiLU backward, pooling, upsampling, the 1x1 output layer,
// the loss, Adam) is plain CUDA-core code.
#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <math.h>
#include <stdint.h>

#include <algorithm>

#include "../../include/lbm_b200.h"
#include "../../include/lbm_surrogate.h"
#include "lbm_shared.h"

namespace lbm {
int set_error(int code, const char *fmt, ...);
extern LaunchCount g_launches;
void *tensor_map_encoder();  // cuTensorMapEncodeTiled, NULL if there is none
}  // namespace lbm

namespace {

typedef __nv_bfloat16 bf16;

constexpr int kThreads = 256;

// Every kernel here but k_conv3x3 is launched as a programmatic dependent of the one before: its
// blocks may be set up while that one still runs, and it reads and writes only
// after dep_sync.  The 118 launches that a training step (batch 16, 128 x 128) then had:
// 1.86 ms as ordinary launches, 1.73 so.
__device__ __forceinline__ void dep_sync()
{
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    asm volatile("griddepcontrol.wait;" ::: "memory");
}

template <typename... KArgs, typename... Args>
void go(void (*k)(KArgs...), dim3 grid, unsigned block, int smem, cudaStream_t s, Args... args)
{
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = dim3(block);
    cfg.dynamicSmemBytes = (size_t)smem;
    cfg.stream = s;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    cudaLaunchKernelEx(&cfg, k, args...);
}

__device__ __forceinline__ void cp_async16(void *smem, const void *gmem, int bytes)
{
    const unsigned s = (unsigned)__cvta_generic_to_shared(smem);
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(s), "l"(gmem), "r"(bytes));
}
__device__ __forceinline__ void cp_commit() { asm volatile("cp.async.commit_group;\n" ::); }
template <int N>
__device__ __forceinline__ void cp_wait()
{
    asm volatile("cp.async.wait_group %0;\n" ::"n"(N));
}

// D += A * B for one 16x8x16 bf16 tile (A row-major, B column-major fragments)
__device__ __forceinline__ void mma16816(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3,
                                         uint32_t b0, uint32_t b1)
{
    asm volatile(
        "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, "
        "{%0,%1,%2,%3};\n"
        : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
        : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

__device__ __forceinline__ uint32_t ld32(const bf16 *p) { return *reinterpret_cast<const uint32_t *>(p); }

__device__ __forceinline__ float silu(float z) { return z / (1.0f + expf(-z)); }
__device__ __forceinline__ float silu_grad(float z)
{
    const float s = 1.0f / (1.0f + expf(-z));
    return s * (1.0f + z * (1.0f - s));
}

// ---------------------------------------------------------------------------
// 3x3 convolution (forward and data gradient)
// ---------------------------------------------------------------------------
constexpr int CBM = 128;       // pixels per block
constexpr int CBK = 32;        // input channels per K chunk (one tap)
constexpr int CLD = CBK + 8;   // shared-memory row stride: rows 80 B apart, conflict-free fragment loads

struct ConvArgs {
    const bf16 *x;
    int64_t xs;
    int xo;
    const bf16 *w;
    const float *bias;
    int B, H, W, Cin, Cout;
    float *of;
    int64_t os;
    int oo, acc;
    bf16 *oa;
    int64_t as;
    int ao, act;
};

// 8 warps: 4 along M (32 pixels each) x 2 along N (BN/2 channels each)
template <int BN>
__global__ void __launch_bounds__(kThreads) k_conv3x3(const ConvArgs a)
{
    dep_sync();
    __shared__ __align__(16) bf16 As[2][CBM * CLD];
    __shared__ __align__(16) bf16 Bs[2][BN * CLD];
    constexpr int NT = BN / 16;  // n8 tiles per warp
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int wm = warp & 3, wn = warp >> 2;
    const int64_t M = (int64_t)a.B * a.H * a.W;
    const int64_t m0 = (int64_t)blockIdx.x * CBM;
    const int n0 = blockIdx.y * BN;
    const int cchunks = a.Cin / CBK;
    const int nk = 9 * cchunks;

    // the two 16-byte pieces of the A tile this thread gathers
    int ar[2], aq[2], ab[2], ay[2], ax[2];
    bool av[2];
#pragma unroll
    for (int i = 0; i < 2; ++i) {
        const int v = tid + i * kThreads;
        ar[i] = v >> 2;
        aq[i] = v & 3;
        const int64_t m = m0 + ar[i];
        av[i] = m < M;
        const int64_t mm = av[i] ? m : 0;
        ax[i] = int(mm % a.W);
        ay[i] = int((mm / a.W) % a.H);
        ab[i] = int(mm / ((int64_t)a.W * a.H));
    }

    auto load = [&](int kc, int st) {
        const int tap = kc / cchunks, c0 = (kc % cchunks) * CBK;
        const int dy = tap / 3 - 1, dx = tap % 3 - 1;
#pragma unroll
        for (int i = 0; i < 2; ++i) {
            const int yy = ay[i] + dy, xx = ax[i] + dx;
            const bool ok = av[i] && yy >= 0 && yy < a.H && xx >= 0 && xx < a.W;
            const bf16 *src =
                ok ? a.x + ((int64_t)(ab[i] * a.H + yy) * a.W + xx) * a.xs + a.xo + c0 + aq[i] * 8 : a.x;
            cp_async16(&As[st][ar[i] * CLD + aq[i] * 8], src, ok ? 16 : 0);
        }
        if (tid < BN * 4) {
            const int r = tid >> 2, q = tid & 3;
            const int n = n0 + r;
            const bool ok = n < a.Cout;
            const bf16 *src = ok ? a.w + ((int64_t)n * 9 + tap) * a.Cin + c0 + q * 8 : a.w;
            cp_async16(&Bs[st][r * CLD + q * 8], src, ok ? 16 : 0);
        }
        cp_commit();
    };

    float acc[2][NT][4];
#pragma unroll
    for (int i = 0; i < 2; ++i)
#pragma unroll
        for (int j = 0; j < NT; ++j)
#pragma unroll
            for (int e = 0; e < 4; ++e) acc[i][j][e] = 0.0f;

    const int g = lane >> 2, t = lane & 3;
    load(0, 0);
    for (int kc = 0; kc < nk; ++kc) {
        const int st = kc & 1;
        if (kc + 1 < nk) {
            load(kc + 1, st ^ 1);
            cp_wait<1>();
        } else {
            cp_wait<0>();
        }
        __syncthreads();
        const bf16 *as_ = As[st];
        const bf16 *bs_ = Bs[st];
#pragma unroll
        for (int ks = 0; ks < CBK; ks += 16) {
            const int col = ks + 2 * t;
            uint32_t af[2][4], bfr[NT][2];
#pragma unroll
            for (int mt = 0; mt < 2; ++mt) {
                const int row = wm * 32 + mt * 16 + g;
                af[mt][0] = ld32(as_ + row * CLD + col);
                af[mt][1] = ld32(as_ + (row + 8) * CLD + col);
                af[mt][2] = ld32(as_ + row * CLD + col + 8);
                af[mt][3] = ld32(as_ + (row + 8) * CLD + col + 8);
            }
#pragma unroll
            for (int nt = 0; nt < NT; ++nt) {
                const int nrow = wn * (BN / 2) + nt * 8 + g;
                bfr[nt][0] = ld32(bs_ + nrow * CLD + col);
                bfr[nt][1] = ld32(bs_ + nrow * CLD + col + 8);
            }
#pragma unroll
            for (int mt = 0; mt < 2; ++mt)
#pragma unroll
                for (int nt = 0; nt < NT; ++nt)
                    mma16816(acc[mt][nt], af[mt][0], af[mt][1], af[mt][2], af[mt][3], bfr[nt][0], bfr[nt][1]);
        }
        __syncthreads();
    }

#pragma unroll
    for (int mt = 0; mt < 2; ++mt)
#pragma unroll
        for (int nt = 0; nt < NT; ++nt)
#pragma unroll
            for (int h = 0; h < 2; ++h)
#pragma unroll
                for (int e = 0; e < 2; ++e) {
                    const int64_t m = m0 + wm * 32 + mt * 16 + g + h * 8;
                    const int n = n0 + wn * (BN / 2) + nt * 8 + 2 * t + e;
                    if (m >= M || n >= a.Cout) continue;
                    float z = acc[mt][nt][h * 2 + e];
                    if (a.bias) z += a.bias[n];
                    if (a.of) {
                        float *p = a.of + m * a.os + a.oo + n;
                        *p = a.acc ? *p + z : z;
                    }
                    if (a.oa) a.oa[m * a.as + a.ao + n] = __float2bfloat16_rn(a.act ? silu(z) : z);
                }
}

__global__ void k_flip(const bf16 *__restrict__ w, bf16 *__restrict__ wt, int Cout, int Cin)
{
    dep_sync();
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    const int64_t n = (int64_t)Cout * 9 * Cin;
    if (i >= n) return;
    // i indexes wt[ci][tap][co]
    const int co = int(i % Cout);
    const int tap = int((i / Cout) % 9);
    const int ci = int(i / ((int64_t)Cout * 9));
    wt[i] = w[((int64_t)co * 9 + (8 - tap)) * Cin + ci];
}

// ---------------------------------------------------------------------------
// sums of the weight gradient's and the column sums' shares
// ---------------------------------------------------------------------------
// out[i] = sum_{s < S} ws[s*n + i] in a fixed order: 32 columns a block, its 32
// warps take every 32nd row and their sums are added in warp order
constexpr int kSumThreads = 1024;
__global__ void __launch_bounds__(kSumThreads) k_sum_splits(const float *__restrict__ ws, int S, int64_t n,
                                                         float *__restrict__ out)
{
    dep_sync();
    __shared__ float sh[kSumThreads / 32][32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int64_t i = (int64_t)blockIdx.x * 32 + lane;
    float s = 0.0f;
    if (i < n) {
        constexpr int ST = kSumThreads / 32;  // rows between a warp's loads
        const float *q = ws + (int64_t)warp * n + i;
        int k = warp;
        for (; k + 7 * ST < S; k += 8 * ST, q += 8 * ST * n) {  // eight loads in flight
            const float v0 = q[0], v1 = q[ST * n], v2 = q[2 * ST * n], v3 = q[3 * ST * n], v4 = q[4 * ST * n],
                        v5 = q[5 * ST * n], v6 = q[6 * ST * n], v7 = q[7 * ST * n];
            s += ((v0 + v1) + (v2 + v3)) + ((v4 + v5) + (v6 + v7));
        }
        for (; k < S; k += ST, q += ST * n) s += *q;
    }
    sh[warp][lane] = s;
    __syncthreads();
    if (warp == 0 && i < n) {
        float tot = sh[0][lane];
#pragma unroll
        for (int k = 1; k < kSumThreads / 32; ++k) tot += sh[k][lane];
        out[i] = tot;
    }
}

// the same for few rows: a thread a column
__global__ void __launch_bounds__(kThreads) k_sum_few(const float *__restrict__ ws, int S, int64_t n,
                                                      float *__restrict__ out)
{
    dep_sync();
    const int64_t i = (int64_t)blockIdx.x * kThreads + threadIdx.x;
    if (i >= n) return;
    const float *q = ws + i;
    float s = 0.0f;
    int k = 0;
    for (; k + 8 <= S; k += 8, q += 8 * n) {
        const float v0 = q[0], v1 = q[n], v2 = q[2 * n], v3 = q[3 * n], v4 = q[4 * n], v5 = q[5 * n], v6 = q[6 * n],
                    v7 = q[7 * n];
        s += ((v0 + v1) + (v2 + v3)) + ((v4 + v5) + (v6 + v7));
    }
    for (; k < S; ++k, q += n) s += *q;
    out[i] = s;
}

// Up to 64 rows a thread has its loads in flight by itself, and the weight
// gradient's partial sums (S n of about 5 M) then have columns for all SMs (10
// rows of 590 K: with the warps along the rows 18 us, so 6).  More rows have
// few columns and need the warps along them (592 rows of 32: 9 us with eight warps, 6 with 32).
void sum_splits(const float *ws, int S, int64_t n, float *out, cudaStream_t s)
{
    if (S <= 64)
        go(k_sum_few, unsigned((n + kThreads - 1) / kThreads), kThreads, 0, s, ws, S, n, out);
    else
        go(k_sum_splits, unsigned((n + 31) / 32), kSumThreads, 0, s, ws, S, n, out);
}

// ---------------------------------------------------------------------------
// column sums (bias gradient) and the SiLU backward pass
// ---------------------------------------------------------------------------
// Both stream a P x C matrix whose only reuse is the column sum: 16-byte loads
// of 8 channels a thread, col_rows(P) rows a block, the threads' sums added in
// shared memory in row order.  Measured at batch 16 of 128^2 images: the SiLU
// backward pass and the column sums of all 14 layers 0.24 + 1.0 ms in two
// scalar passes, 0.15 + 0.11 ms in one.
constexpr int64_t kColBlocks = 592;  // four blocks per SM
// rows per block
__host__ __device__ inline int64_t col_rows(int64_t P)
{
    const int64_t r = (P + kColBlocks - 1) / kColBlocks;
    return r < 16 ? 16 : r;
}

__device__ __forceinline__ void unpack8(const uint4 v, float (&o)[8])
{
    const __nv_bfloat162 *h = reinterpret_cast<const __nv_bfloat162 *>(&v);
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        const float2 f = __bfloat1622float2(h[k]);
        o[2 * k] = f.x;
        o[2 * k + 1] = f.y;
    }
}

__device__ __forceinline__ uint4 pack8(const float (&v)[8])
{
    uint4 o;
    __nv_bfloat162 *h = reinterpret_cast<__nv_bfloat162 *>(&o);
#pragma unroll
    for (int k = 0; k < 4; ++k) h[k] = __floats2bfloat162_rn(v[2 * k], v[2 * k + 1]);
    return o;
}

// a block's rows of 8-channel groups: visit(p, c) for the thread's (row, first
// channel) pairs returns 8 values; their column sums go to ws[blockIdx.x][C]
template <class Visit>
__device__ __forceinline__ void col_block(int64_t P, int C, float *__restrict__ ws, Visit visit)
{
    __shared__ float sh[kThreads * 8];
    const int C8 = C / 8;
    const int64_t nr = col_rows(P), beg = (int64_t)blockIdx.x * nr;
    const int rows = int(beg + nr < P ? nr : P - beg);
    for (int g0 = 0; g0 < C8; g0 += kThreads) {
        const int ng = C8 - g0 < kThreads ? C8 - g0 : kThreads;  // groups of this pass
        const int RL = kThreads / ng;                            // rows side by side
        const int rl = threadIdx.x / ng, g = threadIdx.x % ng;
        float acc[8];
#pragma unroll
        for (int k = 0; k < 8; ++k) acc[k] = 0.0f;
        if (rl < RL)
            for (int r = rl; r < rows; r += RL) {
                float v[8];
                visit(beg + r, (g0 + g) * 8, v);
#pragma unroll
                for (int k = 0; k < 8; ++k) acc[k] += v[k];
            }
        if (ws) {
            if (rl < RL)
#pragma unroll
                for (int k = 0; k < 8; ++k) sh[(rl * ng + g) * 8 + k] = acc[k];
            __syncthreads();
            for (int c = threadIdx.x; c < ng * 8; c += kThreads) {
                float s = 0.0f;
                for (int r = 0; r < RL; ++r) s += sh[r * ng * 8 + c];
                ws[(int64_t)blockIdx.x * C + g0 * 8 + c] = s;
            }
            __syncthreads();
        }
    }
}

__global__ void __launch_bounds__(kThreads) k_colsum8(const bf16 *__restrict__ a, int64_t P, int C,
                                                      float *__restrict__ ws)
{
    dep_sync();
    col_block(P, C, ws, [&](int64_t p, int c, float (&v)[8]) { unpack8(*(const uint4 *)(a + p * C + c), v); });
}

// dz = da * silu'(z) in bf16 and, with ws, the column sums of dz (as rounded)
__global__ void __launch_bounds__(kThreads) k_silu_bwd8(const float *__restrict__ da, int64_t das, int dao,
                                                        const float *__restrict__ z, int64_t P, int C,
                                                        bf16 *__restrict__ dz, float *__restrict__ ws)
{
    dep_sync();
    col_block(P, C, ws, [&](int64_t p, int c, float (&v)[8]) {
        const float4 *d = (const float4 *)(da + p * das + dao + c), *y = (const float4 *)(z + p * C + c);
        const float4 d0 = d[0], d1 = d[1], y0 = y[0], y1 = y[1];
        v[0] = d0.x * silu_grad(y0.x); v[1] = d0.y * silu_grad(y0.y);
        v[2] = d0.z * silu_grad(y0.z); v[3] = d0.w * silu_grad(y0.w);
        v[4] = d1.x * silu_grad(y1.x); v[5] = d1.y * silu_grad(y1.y);
        v[6] = d1.z * silu_grad(y1.z); v[7] = d1.w * silu_grad(y1.w);
        const uint4 q = pack8(v);
        *(uint4 *)(dz + p * C + c) = q;
        unpack8(q, v);
    });
}

// any channel count and alignment
__global__ void __launch_bounds__(kThreads) k_colsum(const bf16 *__restrict__ a, int64_t P, int C,
                                                     float *__restrict__ ws)
{
    dep_sync();
    const int64_t nr = col_rows(P), beg = (int64_t)blockIdx.x * nr;
    const int64_t end = beg + nr < P ? beg + nr : P;
    for (int c = threadIdx.x; c < C; c += kThreads) {
        float s = 0.0f;
        for (int64_t p = beg; p < end; ++p) s += __bfloat162float(a[p * C + c]);
        ws[(int64_t)blockIdx.x * C + c] = s;
    }
}

__global__ void k_silu_bwd(const float *__restrict__ da, int64_t das, int dao, const float *__restrict__ z, int64_t P,
                           int C, bf16 *__restrict__ dz)
{
    dep_sync();
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= P * C) return;
    const int64_t p = i / C;
    const int c = int(i % C);
    dz[i] = __float2bfloat16_rn(da[p * das + dao + c] * silu_grad(z[i]));
}

// ---------------------------------------------------------------------------
// pooling, upsampling, output layer, loss, optimiser
// ---------------------------------------------------------------------------
// The *_v kernels move 16 bytes a thread (8 bf16 or 4 FP32 channels) and take
// one division pair per thread; the plain ones serve channel counts, strides
// and addresses that are no multiple of that.
struct Pix {
    int b, y, x, c;
    bool in;
};
// thread i of a (B, h, w, C) tensor in units of V channels
template <int V>
__device__ __forceinline__ Pix pix_of(int B, int h, int w, int C)
{
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    const int CV = C / V;
    Pix p;
    p.in = i < (int64_t)B * h * w * CV;
    const uint32_t u = uint32_t(i);  // the launch keeps the count below 2^32
    p.c = int(u % CV) * V;
    const uint32_t q = u / CV;
    p.x = int(q % w);
    const uint32_t r = q / w;
    p.y = int(r % h);
    p.b = int(r / h);
    return p;
}

__global__ void __launch_bounds__(kThreads) k_pool2_v(const bf16 *__restrict__ x, int64_t xs, int xo, int B, int H,
                                                      int W, int C, bf16 *__restrict__ y, int64_t ys, int yo)
{
    dep_sync();
    const int h = H / 2, w = W / 2;
    const Pix p = pix_of<8>(B, h, w, C);
    if (!p.in) return;
    const bf16 *s = x + ((int64_t)(p.b * H + 2 * p.y) * W + 2 * p.x) * xs + xo + p.c;
    float a[8], b[8], c[8], d[8], o[8];
    unpack8(*(const uint4 *)s, a);
    unpack8(*(const uint4 *)(s + xs), b);
    unpack8(*(const uint4 *)(s + (int64_t)W * xs), c);
    unpack8(*(const uint4 *)(s + (int64_t)W * xs + xs), d);
#pragma unroll
    for (int k = 0; k < 8; ++k) o[k] = 0.25f * ((a[k] + b[k]) + (c[k] + d[k]));
    *(uint4 *)(y + ((int64_t)(p.b * h + p.y) * w + p.x) * ys + yo + p.c) = pack8(o);
}

__global__ void __launch_bounds__(kThreads) k_up2_v(const bf16 *__restrict__ x, int64_t xs, int xo, int B, int h,
                                                    int w, int C, bf16 *__restrict__ y, int64_t ys, int yo)
{
    dep_sync();
    const Pix p = pix_of<8>(B, h, w, C);
    if (!p.in) return;
    const uint4 v = *(const uint4 *)(x + ((int64_t)(p.b * h + p.y) * w + p.x) * xs + xo + p.c);
    bf16 *o = y + ((int64_t)(p.b * 2 * h + 2 * p.y) * 2 * w + 2 * p.x) * ys + yo + p.c;
    *(uint4 *)o = v;
    *(uint4 *)(o + ys) = v;
    *(uint4 *)(o + (int64_t)2 * w * ys) = v;
    *(uint4 *)(o + (int64_t)2 * w * ys + ys) = v;
}

__global__ void __launch_bounds__(kThreads) k_pool2_bwd_v(const float *__restrict__ dy, int64_t dys, int dyo, int B,
                                                          int H, int W, int C, float *__restrict__ dx, int64_t dxs,
                                                          int dxo)
{
    dep_sync();
    const int h = H / 2, w = W / 2;
    const Pix p = pix_of<4>(B, h, w, C);
    if (!p.in) return;
    const float4 g = *(const float4 *)(dy + ((int64_t)(p.b * h + p.y) * w + p.x) * dys + dyo + p.c);
    float *o = dx + ((int64_t)(p.b * H + 2 * p.y) * W + 2 * p.x) * dxs + dxo + p.c;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        float4 *q = (float4 *)(o + (int64_t)(k >> 1) * W * dxs + (k & 1) * dxs);
        float4 v = *q;
        v.x += 0.25f * g.x; v.y += 0.25f * g.y; v.z += 0.25f * g.z; v.w += 0.25f * g.w;
        *q = v;
    }
}

__global__ void __launch_bounds__(kThreads) k_up2_bwd_v(const float *__restrict__ dy, int64_t dys, int dyo, int B,
                                                        int h, int w, int C, float *__restrict__ dx, int64_t dxs,
                                                        int dxo, int accumulate)
{
    dep_sync();
    const Pix p = pix_of<4>(B, h, w, C);
    if (!p.in) return;
    const float *s = dy + ((int64_t)(p.b * 2 * h + 2 * p.y) * 2 * w + 2 * p.x) * dys + dyo + p.c;
    const float4 a = *(const float4 *)s, b = *(const float4 *)(s + dys);
    const float4 c = *(const float4 *)(s + (int64_t)2 * w * dys), d = *(const float4 *)(s + (int64_t)2 * w * dys + dys);
    float4 r = make_float4((a.x + b.x) + (c.x + d.x), (a.y + b.y) + (c.y + d.y), (a.z + b.z) + (c.z + d.z),
                           (a.w + b.w) + (c.w + d.w));
    float4 *o = (float4 *)(dx + ((int64_t)(p.b * h + p.y) * w + p.x) * dxs + dxo + p.c);
    if (accumulate) {
        const float4 v = *o;
        r.x = v.x + r.x; r.y = v.y + r.y; r.z = v.z + r.z; r.w = v.w + r.w;
    }
    *o = r;
}

__global__ void k_pool2(const bf16 *__restrict__ x, int64_t xs, int xo, int B, int H, int W, int C,
                        bf16 *__restrict__ y, int64_t ys, int yo)
{
    dep_sync();
    const int h = H / 2, w = W / 2;
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= (int64_t)B * h * w * C) return;
    const int c = int(i % C);
    const int64_t q = i / C;
    const int X = int(q % w), Y = int((q / w) % h), b = int(q / ((int64_t)w * h));
    auto at = [&](int yy, int xx) { return __bfloat162float(x[((int64_t)(b * H + yy) * W + xx) * xs + xo + c]); };
    const float s = (at(2 * Y, 2 * X) + at(2 * Y, 2 * X + 1)) + (at(2 * Y + 1, 2 * X) + at(2 * Y + 1, 2 * X + 1));
    y[q * ys + yo + c] = __float2bfloat16_rn(0.25f * s);
}

__global__ void k_pool2_bwd(const float *__restrict__ dy, int64_t dys, int dyo, int B, int H, int W, int C,
                            float *__restrict__ dx, int64_t dxs, int dxo)
{
    dep_sync();
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= (int64_t)B * H * W * C) return;
    const int c = int(i % C);
    const int64_t q = i / C;
    const int xx = int(q % W), yy = int((q / W) % H), b = int(q / ((int64_t)W * H));
    const int64_t src = ((int64_t)(b * (H / 2) + yy / 2) * (W / 2) + xx / 2) * dys + dyo + c;
    dx[q * dxs + dxo + c] += 0.25f * dy[src];
}

__global__ void k_up2(const bf16 *__restrict__ x, int64_t xs, int xo, int B, int h, int w, int C,
                      bf16 *__restrict__ y, int64_t ys, int yo)
{
    dep_sync();
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    const int H = 2 * h, W = 2 * w;
    if (i >= (int64_t)B * H * W * C) return;
    const int c = int(i % C);
    const int64_t q = i / C;
    const int X = int(q % W), Y = int((q / W) % H), b = int(q / ((int64_t)W * H));
    y[q * ys + yo + c] = x[((int64_t)(b * h + Y / 2) * w + X / 2) * xs + xo + c];
}

__global__ void k_up2_bwd(const float *__restrict__ dy, int64_t dys, int dyo, int B, int h, int w, int C,
                          float *__restrict__ dx, int64_t dxs, int dxo, int accumulate)
{
    dep_sync();
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= (int64_t)B * h * w * C) return;
    const int c = int(i % C);
    const int64_t q = i / C;
    const int X = int(q % w), Y = int((q / w) % h), b = int(q / ((int64_t)w * h));
    const int W = 2 * w, H = 2 * h;
    auto at = [&](int yy, int xx) { return dy[((int64_t)(b * H + yy) * W + xx) * dys + dyo + c]; };
    const float s = (at(2 * Y, 2 * X) + at(2 * Y, 2 * X + 1)) + (at(2 * Y + 1, 2 * X) + at(2 * Y + 1, 2 * X + 1));
    float *o = dx + q * dxs + dxo + c;
    *o = accumulate ? *o + s : s;
}

constexpr int kMaxJ = 8;

__global__ void k_head(const bf16 *__restrict__ a, int64_t as, int ao, const bf16 *__restrict__ wh,
                       const float *__restrict__ bh, int64_t P, int C, int J, float *__restrict__ y)
{
    dep_sync();
    const int64_t p = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= P) return;
    float acc[kMaxJ];
    for (int j = 0; j < J; ++j) acc[j] = bh ? bh[j] : 0.0f;
    for (int c = 0; c < C; ++c) {
        const float v = __bfloat162float(a[p * as + ao + c]);
        for (int j = 0; j < J; ++j) acc[j] += v * __bfloat162float(wh[j * C + c]);
    }
    for (int j = 0; j < J; ++j) y[p * J + j] = acc[j];
}

__global__ void k_head_bwd_da(const float *__restrict__ dy, const bf16 *__restrict__ wh, int64_t P, int C, int J,
                              float *__restrict__ da, int64_t das, int dao)
{
    dep_sync();
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= P * C) return;
    const int64_t p = i / C;
    const int c = int(i % C);
    float s = 0.0f;
    for (int j = 0; j < J; ++j) s += dy[p * J + j] * __bfloat162float(wh[j * C + c]);
    da[p * das + dao + c] = s;
}

// the network's own head: three outputs, channels in multiples of 8
__global__ void __launch_bounds__(kThreads) k_head3_v(const bf16 *__restrict__ a, int64_t as, int ao,
                                                      const bf16 *__restrict__ wh, const float *__restrict__ bh,
                                                      int64_t P, int C, float *__restrict__ y)
{
    dep_sync();
    const int64_t p = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= P) return;
    float acc[3];
    for (int j = 0; j < 3; ++j) acc[j] = bh ? bh[j] : 0.0f;
    for (int c = 0; c < C; c += 8) {
        float v[8];
        unpack8(*(const uint4 *)(a + p * as + ao + c), v);
#pragma unroll
        for (int k = 0; k < 8; ++k)
#pragma unroll
            for (int j = 0; j < 3; ++j) acc[j] += v[k] * __bfloat162float(wh[j * C + c + k]);
    }
    for (int j = 0; j < 3; ++j) y[p * 3 + j] = acc[j];
}

__global__ void __launch_bounds__(kThreads) k_head3_bwd_da_v(const float *__restrict__ dy, const bf16 *__restrict__ wh,
                                                             int64_t P, int C, float *__restrict__ da, int64_t das,
                                                             int dao)
{
    dep_sync();
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    const int C4 = C / 4;
    if (i >= P * C4) return;
    const int64_t p = i / C4;
    const int c = int(i % C4) * 4;
    const float d[3] = {dy[p * 3], dy[p * 3 + 1], dy[p * 3 + 2]};
    float s[4] = {0.0f, 0.0f, 0.0f, 0.0f};
#pragma unroll
    for (int j = 0; j < 3; ++j)
#pragma unroll
        for (int k = 0; k < 4; ++k) s[k] += d[j] * __bfloat162float(wh[j * C + c + k]);
    *(float4 *)(da + p * das + dao + c) = make_float4(s[0], s[1], s[2], s[3]);
}

constexpr int64_t kHeadRows = 512;

// per pixel range: items j*C + c (dwh) and J*C + j (dbh); 32 channels x 8 rows
// side by side, the row sums added in row order
__global__ void __launch_bounds__(kThreads) k_head_bwd_w(const float *__restrict__ dy, const bf16 *__restrict__ a,
                                                         int64_t as, int ao, int64_t P, int C, int J,
                                                         float *__restrict__ ws)
{
    dep_sync();
    __shared__ float sh[kThreads / 32][kMaxJ][33];
    const int lane = threadIdx.x & 31, rl = threadIdx.x >> 5;
    const int items = J * C + J;
    const int64_t beg = (int64_t)blockIdx.x * kHeadRows;
    const int64_t end = beg + kHeadRows < P ? beg + kHeadRows : P;
    float *o = ws + (int64_t)blockIdx.x * items;
    // one column past the channels stands for the constant 1 (dbh)
    for (int cb = 0; cb <= C; cb += 32) {
        const int c = cb + lane;
        float acc[kMaxJ];
#pragma unroll
        for (int j = 0; j < kMaxJ; ++j) acc[j] = 0.0f;
        if (c <= C)
            for (int64_t p = beg + rl; p < end; p += kThreads / 32) {
                const float v = c < C ? __bfloat162float(a[p * as + ao + c]) : 1.0f;
#pragma unroll
                for (int j = 0; j < kMaxJ; ++j)
                    if (j < J) acc[j] += dy[p * J + j] * v;
            }
#pragma unroll
        for (int j = 0; j < kMaxJ; ++j) sh[rl][j][lane] = acc[j];
        __syncthreads();
        for (int j = rl; j < J; j += kThreads / 32) {
            float s = 0.0f;
            for (int r = 0; r < kThreads / 32; ++r) s += sh[r][j][lane];
            if (c < C) o[j * C + c] = s;
            else if (c == C) o[J * C + j] = s;
        }
        __syncthreads();
    }
}

// the same for the network's own head (J = 3, 8 | C <= 256): 8 channels a thread
__global__ void __launch_bounds__(kThreads) k_head3_bwd_w_v(const float *__restrict__ dy, const bf16 *__restrict__ a,
                                                            int64_t as, int ao, int64_t P, int C,
                                                            float *__restrict__ ws)
{
    dep_sync();
    __shared__ float sh[kThreads * 8], shd[kThreads];
    const int C8 = C / 8, RL = kThreads / C8, rl = threadIdx.x / C8, g = threadIdx.x % C8;
    const int64_t beg = (int64_t)blockIdx.x * kHeadRows;
    const int rows = int(beg + kHeadRows < P ? kHeadRows : P - beg);
    float acc[3][8], accd[3];
#pragma unroll
    for (int j = 0; j < 3; ++j) {
        accd[j] = 0.0f;
#pragma unroll
        for (int k = 0; k < 8; ++k) acc[j][k] = 0.0f;
    }
    if (rl < RL)
#pragma unroll 2
        for (int r = rl; r < rows; r += RL) {
            const int64_t p = beg + r;
            float v[8];
            unpack8(*(const uint4 *)(a + p * as + ao + g * 8), v);
#pragma unroll
            for (int j = 0; j < 3; ++j) {
                const float d = dy[p * 3 + j];
                accd[j] += d;
#pragma unroll
                for (int k = 0; k < 8; ++k) acc[j][k] += d * v[k];
            }
        }
    float *o = ws + (int64_t)blockIdx.x * (3 * C + 3);
#pragma unroll
    for (int j = 0; j < 3; ++j) {
        if (rl < RL) {
#pragma unroll
            for (int k = 0; k < 8; ++k) sh[(rl * C8 + g) * 8 + k] = acc[j][k];
            if (g == 0) shd[rl] = accd[j];
        }
        __syncthreads();
        for (int c = threadIdx.x; c <= C; c += kThreads) {
            float s = 0.0f;
            for (int r = 0; r < RL; ++r) s += c < C ? sh[r * C + c] : shd[r];
            o[c < C ? j * C + c : 3 * C + j] = s;
        }
        __syncthreads();
    }
}

constexpr int kMseBlocks = 296;

__global__ void k_mse(const float *__restrict__ y, const float *__restrict__ t, const float *__restrict__ cw, int64_t P,
                      int J, float *__restrict__ dy, float *__restrict__ ws)
{
    dep_sync();
    __shared__ float sh[kThreads / 32];
    const int64_t n = P * J;
    const float inv = 1.0f / float(n);
    float s = 0.0f;
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        const int j = int(i % J);
        const float d = y[i] - t[i];
        const float w = cw ? cw[j] : 1.0f;
        dy[i] = 2.0f * w * d * inv;
        s += w * d * d;
    }
    for (int o = 16; o > 0; o >>= 1) s += __shfl_down_sync(0xffffffffu, s, o);
    if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = s;
    __syncthreads();
    if (threadIdx.x == 0) {
        float tot = 0.0f;
        for (int k = 0; k < kThreads / 32; ++k) tot += sh[k];
        ws[blockIdx.x] = tot;
    }
}

__global__ void k_mse_final(const float *__restrict__ ws, int nb, int64_t n, float *__restrict__ loss)
{
    dep_sync();
    float s = 0.0f;  // one warp: lane l takes every 32nd block's sum, then a fixed tree
    for (int k = threadIdx.x; k < nb; k += 32) s += ws[k];
    for (int o = 16; o > 0; o >>= 1) s += __shfl_down_sync(0xffffffffu, s, o);
    if (threadIdx.x == 0) *loss = s / float(n);
}

__global__ void k_adam(float *__restrict__ p, bf16 *__restrict__ pb, const float *__restrict__ g, float *__restrict__ m,
                       float *__restrict__ v, int64_t n, float lr, float b1, float b2, float eps, float c1, float c2,
                       float wd)
{
    dep_sync();
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const float gi = g[i];
    const float mi = b1 * m[i] + (1.0f - b1) * gi;
    const float vi = b2 * v[i] + (1.0f - b2) * gi * gi;
    m[i] = mi;
    v[i] = vi;
    const float pi = p[i] - lr * ((mi / c1) / (sqrtf(vi / c2) + eps) + wd * p[i]);
    p[i] = pi;
    if (pb) pb[i] = __float2bfloat16_rn(pi);
}

__global__ void k_to_bf16(const float *__restrict__ x, bf16 *__restrict__ y, int64_t n)
{
    dep_sync();
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) y[i] = __float2bfloat16_rn(x[i]);
}

unsigned blocks_for(int64_t n) { return unsigned((n + kThreads - 1) / kThreads); }

int launched(const char *what, int count = 1)
{
    lbm::g_launches += count;
    const cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return lbm::set_error(LBM_ERR_CUDA, "%s: %s", what, cudaGetErrorString(e));
    return LBM_OK;
}

bool aligned16(const void *p) { return ((uintptr_t)p & 15u) == 0; }

// ---------------------------------------------------------------------------
// 3x3 convolution on the 5th-generation tensor cores (tcgen05, TMEM)
// ---------------------------------------------------------------------------
// The implicit GEMM of k_conv3x3 (M = pixels, N = Cout, K = 9 Cin) on a tile of
// 8 x 16 pixels, with the accumulators (128 pixels x BN channels, FP32) in tensor
// memory.  The kernel was bound by gathering the im2col matrix, nine copies of
// every pixel; here a K chunk is 32 input channels and all nine
// taps, and its pixels are staged once, with a one-pixel border:
//   * A lies as rows of one pixel's 32 channels, 64 bytes under the 64-byte swizzle,
//     18 x 10 of them.  The 8 pixels of a tile row are a core matrix, the rows of
//     the tile 640 bytes apart (stride offset); the swizzle goes by address bits, so
//     a tap is a shift of the start address by whole pixels;
//   * B is the chunk's weights of the nine taps, [tap][BN][64 bytes], likewise;
//   * rows of 64 bytes are what the copies want: a TMA box costs about 1.2 cycles a
//     row whatever its length, and rows of 16 bytes (8 channels, no swizzle) made
//     the copies the bottleneck.  us at batch 16, 16-byte rows -> 64: 64 -> 64 channels at
//     64 x 64 29 -> 14, 192 -> 64 50 -> 22, 32 -> 32 at 128 x 128 34 -> 21;
//   * one thread issues the copies, one TMA box for a tile's pixels (zero outside
//     the image) and one for the weights, another a chunk's 18 tcgen05.mma (K =
//     16), committed to the stage's mbarrier; copies by all threads took 2000 cycles
//     a chunk for their addresses, and the MMAs' descriptors, computed anew for
//     each, 130 cycles an MMA (us, so and as constants: 384 -> 128 at 32 x 32,
//     batch 1, 16.5 -> 11.3; 256 -> 256 at 16 x 16 12.4 -> 8.9);
//   * the launch is a programmatic dependent: its set-up overlaps the end of the
//     kernel before;
//   * the epilogue reads the accumulators with tcgen05.ld, a thread one pixel and
//     16 channels at a time, and stores whole 32-byte sectors.
// Measured at batch 16 of 128^2 images, all 27 forward and data-gradient layers of
// a training step: mma.sync kernel 1.64 ms, with copies by all threads 1.01 ms,
// this kernel 0.54 ms; 256 -> 256 at 16 x 16, batch 1: 53, 24 and 8.9 us.
// Every mbarrier wait is bounded; on timeout the CTA counts the event in
// g_nn_timeouts (read by lbm_nn_timeouts), waits (bounded) for its own copies and
// MMAs, stores NaN in place of its results, so that nothing downstream takes what an
// earlier call left there for an answer, frees its tensor memory and returns.
constexpr int TBM = 128, TBK = 32, TTHREADS = 256;
constexpr int TTW = 8, TTH = 16, THW = TTW + 2, THP = THW * (TTH + 2);  // pixel tile, its border, their pixels
constexpr long long kNnWaitCycles = 2000000000LL;  // ~1 s at 1.9 GHz
__device__ int g_nn_timeouts;
__device__ long long g_nn_wait_limit = kNnWaitCycles;  // lbm_nn_set_wait_limit

__device__ __forceinline__ uint32_t smem_u32(const void *p) { return (uint32_t)__cvta_generic_to_shared(p); }

__device__ __forceinline__ void nn_mbar_init(uint64_t *b, uint32_t n)
{
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(b)), "r"(n) : "memory");
}

// a wait suspends the thread until the phase completes, `hint` ns at most
__device__ __forceinline__ bool nn_mbar_test(uint64_t *b, uint32_t parity, uint32_t hint)
{
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2, %3;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}\n"
        : "=r"(ok)
        : "r"(smem_u32(b)), "r"(parity), "r"(hint)
        : "memory");
    return ok != 0;
}

__device__ __forceinline__ bool nn_mbar_wait(uint64_t *b, uint32_t parity, long long limit = kNnWaitCycles)
{
    const uint32_t hint = limit < kNnWaitCycles ? 1u : 1000000u;  // short limits must be able to run out (tests)
    if (nn_mbar_test(b, parity, hint)) return true;
    const long long t0 = clock64();
    while (!nn_mbar_test(b, parity, hint))
        if (clock64() - t0 > limit) return false;
    return true;
}

// a block that gave up: the last `stages` of the `copies` its copying thread (tid 32) issued, and the MMAs of the
// `chunks` its issuing thread (tid 0) committed, end before the memory they use is released
__device__ __forceinline__ void nn_drain(int tid, uint64_t *full, uint64_t *bars, int stages, int copies, int chunks)
{
    if (tid == 32)
        for (int k = copies > stages ? copies - stages : 0; k < copies; ++k)
            nn_mbar_wait(&full[k % stages], uint32_t((k / stages) & 1));
    if (tid == 0) {
        if (chunks > 0) nn_mbar_wait(&bars[(chunks - 1) % stages], uint32_t(((chunks - 1) / stages) & 1));
        atomicAdd(&g_nn_timeouts, 1);
    }
    __syncthreads();
}

__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }

// shared-memory matrix descriptor: start address, byte offset of the next 8 rows
// (both >> 4), descriptor version 1, base offset 0, rows of 64 bytes, 64-byte swizzle
__device__ __forceinline__ uint64_t umma_desc(uint32_t addr, uint32_t sbo)
{
    return (uint64_t)((addr >> 4) & 0x3FFFu) | ((uint64_t)1 << 16) | ((uint64_t)((sbo >> 4) & 0x3FFFu) << 32) |
           ((uint64_t)1 << 46) | ((uint64_t)4 << 61);
}

// instruction descriptor of kind::f16: FP32 accumulator, bf16 A and B, both
// K-major, N = BN, M = 128
template <int BN>
__host__ __device__ constexpr uint32_t umma_idesc()
{
    return (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(BN >> 3) << 17) | ((uint32_t)(TBM >> 4) << 24);
}

template <int BN>
struct TcLayout {
    static constexpr int ROW = TBK * 2;                // 64: a pixel's, an output channel's input channels
    static constexpr int A_TX = THP * ROW;             // the tile and its border
    static constexpr int A_BYTES = (A_TX + 1023) / 1024 * 1024;
    static constexpr int TAP = BN * ROW;               // a tap's weights
    static constexpr int BOFF = A_BYTES;
    static constexpr int STAGE = BOFF + 9 * TAP;
    static constexpr int HEAD = 1024;                  // mbarriers, the TMEM address, the channels' bias
    static_assert(STAGE % 1024 == 0 && 128 + BN * 4 <= HEAD, "the swizzle goes by address bits");
    static constexpr int COLS = BN;                    // TMEM columns
    static_assert(COLS == 32 || COLS == 64, "TMEM allocations are powers of two >= 32");
    static constexpr int smem(int stages) { return HEAD + stages * STAGE + 1024; }
    // shared memory bounds the CTAs per SM, so their TMEM columns fit the SM's 512
    static_assert((228 * 1024 / smem(1)) * COLS <= 512, "TMEM oversubscription");
};

__device__ __forceinline__ void st_v8(float *p, const float *v)
{
    asm volatile("st.global.v8.f32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};" ::"l"(p), "f"(v[0]), "f"(v[1]), "f"(v[2]),
                 "f"(v[3]), "f"(v[4]), "f"(v[5]), "f"(v[6]), "f"(v[7])
                 : "memory");
}

__device__ __forceinline__ void nn_expect(uint64_t *b, uint32_t bytes)
{
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(b)), "r"(bytes) : "memory");
}

__device__ __forceinline__ void nn_tma3(void *dst, const CUtensorMap *m, uint64_t *bar, int c0, int c1, int c2)
{
    asm volatile(
        "cp.async.bulk.tensor.3d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], "
        "[%5];" ::"r"(smem_u32(dst)), "l"(m), "r"(c0), "r"(c1), "r"(c2), "r"(smem_u32(bar))
        : "memory");
}

__device__ __forceinline__ void nn_tma4(void *dst, const CUtensorMap *m, uint64_t *bar, int c0, int c1, int c2, int c3)
{
    asm volatile(
        "cp.async.bulk.tensor.4d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4, %5}], "
        "[%6];" ::"r"(smem_u32(dst)), "l"(m), "r"(c0), "r"(c1), "r"(c2), "r"(c3), "r"(smem_u32(bar))
        : "memory");
}

// the same for a channel-major operand: mn, k: byte offsets of the next 32 channels and of the next 8 rows
__device__ __forceinline__ uint64_t wg_desc(uint32_t addr, uint32_t mn, uint32_t k)
{
    return (uint64_t)((addr >> 4) & 0x3FFFu) | ((uint64_t)((mn >> 4) & 0x3FFFu) << 16) |
           ((uint64_t)((k >> 4) & 0x3FFFu) << 32) | ((uint64_t)1 << 46) | ((uint64_t)4 << 61);
}

// 16 accumulator columns of the warp's 32 lanes
__device__ __forceinline__ void tmem_ld16(uint32_t addr, uint32_t (&r)[16])
{
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
          "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
        : "r"(addr)
        : "memory");
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
}

// vec: the outputs' channel strides, offsets and addresses allow 32-byte stores
template <int BN, int NST>
__global__ void __launch_bounds__(TTHREADS)
k_conv3x3_tc(const ConvArgs a, const __grid_constant__ CUtensorMap xmap, const __grid_constant__ CUtensorMap wmap, int ntx,
             int nty, int vec)
{
    using Lt = TcLayout<BN>;
    extern __shared__ unsigned char tc_raw[];
    unsigned char *sm = tc_raw + ((1024u - (smem_u32(tc_raw) & 1023u)) & 1023u);
    uint64_t *full = reinterpret_cast<uint64_t *>(sm);  // a stage's copies have landed
    uint64_t *bars = full + NST;                        // the MMAs that read it are complete
    uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(bars + NST);
    float *sbias = reinterpret_cast<float *>(sm + 128);
    unsigned char *stages = sm + Lt::HEAD;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int n0 = blockIdx.y * BN;
    const int nk = a.Cin / TBK;
    const long long limit = g_nn_wait_limit;

    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)),
                     "r"(Lt::COLS)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    if (tid == 0) {
        for (int k = 0; k < NST; ++k) {
            nn_mbar_init(&full[k], 1);
            nn_mbar_init(&bars[k], 1);
        }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    }
    if (tid == 32) {
        asm volatile("prefetch.tensormap [%0];" ::"l"(&xmap) : "memory");
        asm volatile("prefetch.tensormap [%0];" ::"l"(&wmap) : "memory");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = *tmem_slot;
    // only now that this block has its tensor memory: a dependent's block that took it first would wait for this grid
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    asm volatile("griddepcontrol.wait;" ::: "memory");  // from here on: what earlier kernels wrote
    if (tid >= 64 && tid - 64 < BN)  // read after the next block barrier
        sbias[tid - 64] = a.bias && n0 + tid - 64 < a.Cout ? a.bias[n0 + tid - 64] : 0.0f;

    constexpr uint32_t idesc = umma_idesc<BN>();
    bool fail = false;
    int kc = 0;  // chunks this thread has issued
    if (tid == 32) {  // the copies
        for (; kc < nk; ++kc) {
            const int st = kc % NST;
            if (kc >= NST && !nn_mbar_wait(&bars[st], uint32_t((kc / NST - 1) & 1), limit)) {
                fail = true;
                break;
            }
            unsigned char *base = stages + st * Lt::STAGE;
            const int t = blockIdx.x;
            nn_expect(&full[st], uint32_t(Lt::A_TX + 9 * Lt::TAP));
            nn_tma4(base, &xmap, &full[st], kc * TBK, (t % ntx) * TTW - 1, ((t / ntx) % nty) * TTH - 1,
                    t / (ntx * nty));
            nn_tma3(base + Lt::BOFF, &wmap, &full[st], kc * TBK, n0, 0);
        }
    } else if (tid == 0) {  // the MMAs
        for (; kc < nk; ++kc) {
            if (!nn_mbar_wait(&full[kc % NST], uint32_t((kc / NST) & 1), limit)) {
                fail = true;
                break;
            }
            tc_fence_after();
            // a descriptor's address field counts 16 bytes: a tap or 16 channels on is a constant more
            const uint32_t base = smem_u32(stages + (kc % NST) * Lt::STAGE);
            const uint64_t da0 = umma_desc(base, THW * Lt::ROW), db0 = umma_desc(base + Lt::BOFF, 8 * Lt::ROW);
#pragma unroll
            for (int tap = 0; tap < 9; ++tap) {
#pragma unroll
                for (int ks = 0; ks < TBK; ks += 16) {
                    const uint64_t da = da0 + (uint64_t)(((tap / 3) * THW + tap % 3) * Lt::ROW + ks * 2) / 16;
                    const uint64_t db = db0 + (uint64_t)(tap * Lt::TAP + ks * 2) / 16;
                    const uint32_t accum = tap > 0 || ks > 0 ? 1u : uint32_t(kc > 0);
                    asm volatile(
                        "{\n\t.reg .pred p;\n\t"
                        "setp.ne.b32 p, %4, 0;\n\t"
                        "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}\n" ::"r"(tmem),
                        "l"(da), "l"(db), "r"(idesc), "r"(accum)
                        : "memory");
                }
            }
            asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(
                             smem_u32(&bars[kc % NST]))
                         : "memory");
        }
    }
    __syncwarp();
    // every MMA of this CTA is complete once the commit of the last chunk arrives
    // (for tid 0, which has seen the stage's earlier use complete; the others go by the block barrier)
    const bool done = nn_mbar_wait(&bars[(nk - 1) % NST], uint32_t(((nk - 1) / NST) & 1), limit);
    const bool bad = __syncthreads_or(fail || !done);
    tc_fence_after();
    if (bad) nn_drain(tid, full, bars, NST, kc, kc);
    {
        // warp w reads TMEM lanes 32 (w % 4) ..: pixels 4 tile rows; two warpgroups split the channel slices
        const int wg = warp >> 2;
        const int t = blockIdx.x;
        const int row = (warp & 3) * 32 + lane;
        const int xx = (t % ntx) * TTW + (row & 7), yy = ((t / ntx) % nty) * TTH + (row >> 3), b = t / (ntx * nty);
        const bool px = xx < a.W && yy < a.H;
        const int64_t m = ((int64_t)b * a.H + yy) * a.W + xx;
#pragma unroll 1
        for (int sl = wg; sl < BN / 16; sl += 2) {
            uint32_t r[16];
            tmem_ld16(tmem + ((uint32_t)((warp & 3) * 32) << 16) + (uint32_t)(sl * 16), r);
            const int n = n0 + sl * 16;
            if (!px || n >= a.Cout) continue;
            float z[16];
#pragma unroll
            for (int j = 0; j < 16; ++j) z[j] = __uint_as_float(r[j]) + sbias[sl * 16 + j];
            if (bad)
#pragma unroll
                for (int j = 0; j < 16; ++j) z[j] = NAN;
            if (vec && n + 16 <= a.Cout) {
                if (a.of) {
                    float *p = a.of + m * a.os + a.oo + n;
                    st_v8(p, z);
                    st_v8(p + 8, z + 8);
                }
                if (a.oa) {
                    float h[8];
#pragma unroll
                    for (int j = 0; j < 16; j += 2) {
                        const __nv_bfloat162 v = a.act ? __floats2bfloat162_rn(silu(z[j]), silu(z[j + 1]))
                                                       : __floats2bfloat162_rn(z[j], z[j + 1]);
                        h[j / 2] = *reinterpret_cast<const float *>(&v);
                    }
                    st_v8(reinterpret_cast<float *>(a.oa + m * a.as + a.ao + n), h);
                }
            } else {
#pragma unroll
                for (int j = 0; j < 16; ++j) {
                    if (n + j >= a.Cout) break;
                    if (a.of) {
                        float *p = a.of + m * a.os + a.oo + n + j;
                        *p = a.acc ? *p + z[j] : z[j];
                    }
                    if (a.oa) a.oa[m * a.as + a.ao + n + j] = __float2bfloat16_rn(a.act ? silu(z[j]) : z[j]);
                }
            }
        }
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 0)
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(Lt::COLS) : "memory");
}

// the input as (channel, x, y, image): a box is a tile with its border, zero outside the image; the weights as
// (input channel, output channel, tap)
bool conv_maps(const ConvArgs &a, int BN, CUtensorMap *xm, CUtensorMap *wm)
{
    typedef CUresult (*Encode)(CUtensorMap *, CUtensorMapDataType, cuuint32_t, void *, const cuuint64_t *,
                               const cuuint64_t *, const cuuint32_t *, const cuuint32_t *, CUtensorMapInterleave,
                               CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
    const Encode enc = (Encode)lbm::tensor_map_encoder();
    if (!enc) return false;
    const cuuint32_t one[4] = {1, 1, 1, 1};
    const cuuint64_t row = (cuuint64_t)a.xs * 2;
    const cuuint64_t xd[4] = {(cuuint64_t)a.Cin, (cuuint64_t)a.W, (cuuint64_t)a.H, (cuuint64_t)a.B};
    const cuuint64_t xst[3] = {row, row * a.W, row * a.W * a.H};
    const cuuint32_t xb[4] = {TBK, THW, TTH + 2, 1};
    const cuuint64_t wd[3] = {(cuuint64_t)a.Cin, (cuuint64_t)a.Cout, 9};
    const cuuint64_t wst[2] = {(cuuint64_t)a.Cin * 18, (cuuint64_t)a.Cin * 2};
    const cuuint32_t wb[3] = {TBK, (cuuint32_t)BN, 9};
    return enc(xm, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 4, (void *)(a.x + a.xo), xd, xst, xb, one,
               CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_64B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
               CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS &&
           enc(wm, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, (void *)a.w, wd, wst, wb, one, CU_TENSOR_MAP_INTERLEAVE_NONE,
               CU_TENSOR_MAP_SWIZZLE_64B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) ==
               CUDA_SUCCESS;
}

template <int BN, int NST>
bool launch_conv_tc(const ConvArgs &a, int vec, cudaStream_t s)
{
    using Lt = TcLayout<BN>;
    CUtensorMap xm, wm;
    if (!conv_maps(a, BN, &xm, &wm)) return false;
    const int ntx = (a.W + TTW - 1) / TTW, nty = (a.H + TTH - 1) / TTH;
    cudaFuncSetAttribute(k_conv3x3_tc<BN, NST>, cudaFuncAttributeMaxDynamicSharedMemorySize, Lt::smem(NST));
    const dim3 grid(unsigned(a.B * ntx * nty), unsigned((a.Cout + BN - 1) / BN));
    go(k_conv3x3_tc<BN, NST>, grid, TTHREADS, Lt::smem(NST), s, a, xm, wm, ntx, nty, vec);
    return true;
}

int64_t tc_tiles(const ConvArgs &a) { return (int64_t)a.B * ((a.W + TTW - 1) / TTW) * ((a.H + TTH - 1) / TTH); }

// Channels per block and stages of the ring.  Few blocks are bound by the latency
// of one block's chunks: as many blocks as there are SMs for, and stages that fill
// an SM's shared memory, so that the next kernel's blocks, set up early, don't
// crowd onto some of the SMs (us, 32 channels and 4 / 3 / 2 stages: 128 -> 128 at
// 32 x 32, batch 1, 32 blocks, 6.5 / 7.3 / 7.3; 64 -> 64 at 64 x 64, batch 4, 256 blocks,
// - / 6.6 / 8.1).  More blocks than two an SM take 64 channels, which halves the reads of the
// pixels: up to 296 of those with two stages (64 -> 128 at 32 x 32, batch 16, 256
// blocks: two 8.9, one 13.2, three 13 and more), beyond it with one, where four
// blocks an SM overlap one another (64 -> 64 at 64 x 64, batch 16, 512 blocks: one
// 13.5, two 16.3; 32 channels a block 17.3; 128 -> 384 at 32 x 32: 64 channels 27, 128 31).
// Two tiles a block that share the weights gain nothing (32 -> 32 at 128 x 128: 28.8 against 23.8).
bool conv_tc(const ConvArgs &a, cudaStream_t s)
{
    const int64_t tiles = tc_tiles(a);
    const auto ok32 = [](const void *p) { return ((uintptr_t)p & 31u) == 0; };
    const int vec = !a.acc && (!a.of || ((a.os | a.oo) % 8 == 0 && ok32(a.of))) &&
                    (!a.oa || ((a.as | a.ao) % 16 == 0 && ok32(a.oa)));
    const int64_t n64 = tiles * ((a.Cout + 63) / 64), n32 = tiles * ((a.Cout + 31) / 32);
    if (n32 <= 148) return launch_conv_tc<32, 4>(a, vec, s);
    if (n32 <= 296) return launch_conv_tc<32, 3>(a, vec, s);
    if (a.Cout <= 32) return launch_conv_tc<32, 1>(a, vec, s);
    return n64 <= 296 ? launch_conv_tc<64, 2>(a, vec, s) : launch_conv_tc<64, 1>(a, vec, s);
}

// ---------------------------------------------------------------------------
// 3x3 weight gradient on the 5th-generation tensor cores
// ---------------------------------------------------------------------------
// dw[co][tap][ci] = sum_p dz[p][co] x[p + offset(tap)][ci]: M = 128 output channels,
// N = 32 input channels x 9 taps, K = pixels, a block's share of the pixel tiles
// after one another.  dz and x lie as in the convolution, rows of 32
// channels under the 64-byte swizzle, a tile's dz as [32 channels][128 pixels], its
// x with the border; both operands are channel-major (their K runs over the
// rows).  A step of 16 pixels is two tile rows.  The next 32 columns of B are the
// same channels a pixel further right, so one MMA takes the three taps of a tap row
// (96 columns); the three tap rows have accumulators of their own, 288 columns.
// Fewer than 128 output channels leave rows of the accumulators unused; their part
// of A is never loaded.  The shares' partial sums are added in a fixed order.
// Measured, us with that sum, mma.sync kernel -> this: 32 -> 32 channels at 128 x 128,
// batch 16, 27.9 -> 20.9, 96 -> 32 64 -> 50, 384 -> 128 at 32 x 32 74 -> 21, 256 -> 256 at 16 x 16
// 27.8 -> 14.0; batch 1: 13.6 -> 6.5, -, 14.6 -> 9.9, 10.2 -> 10.5; 256 images of 4 x 4, 256
// channels 109 -> 26.  A training step's 14 layers 0.46 -> 0.25 ms.  Where channels are few
// the tiles' 128 rows of A are mostly unused and the MMAs (24 a tile) are the
// bound; at batch 1 the launch, one tile's latency and the sum.  Against 64-bit
// sums the error is 1e-7 to 6e-6 of the result, as long as a share's chain.
//
// A tile that reaches past the image multiplies zeros of dz by x, and next to the
// border that is an x of the image: the pixel right of the last column meets it in
// the taps to the left, the row below the last one in the taps above.  An
// infinity there must not turn into a NaN of taps that don't use it (RAG): tiles at
// the right edge take the left taps from a second copy of x without the last column,
// and a step whose second row is outside takes that row's x from zeros.
constexpr int WCOLS = 512;                          // TMEM columns (a power of two)
constexpr int WA_ATOM = TBM * 64, WA = 4 * WA_ATOM;  // dz: 32 channels of a tile, all
constexpr int WX_TX = THP * 64, WX = (WX_TX + 1023) / 1024 * 1024;
constexpr int WZERO = (8 + 2) * 64;                 // a row of x with its border
template <bool RAG>
struct WgLayout {
    static constexpr int ST = RAG ? 3 : 4;          // stages
    static constexpr int STAGE = WA + (RAG ? 2 : 1) * WX, ZERO = 1024 + ST * STAGE;
    static constexpr int SMEM = ZERO + (RAG ? 1024 : 0) + 1024;
    static_assert(WZERO <= 1024 && SMEM <= 227 * 1024 && ST * STAGE < (1 << 18), "strides have 14 bits of 16 bytes");
};

// FP32 accumulators, bf16 A and B, both channel-major, M = 128, N
__host__ __device__ constexpr uint32_t wg_idesc(int N)
{
    return (1u << 4) | (1u << 7) | (1u << 10) | (1u << 15) | (1u << 16) | ((uint32_t)(N >> 3) << 17) | (8u << 24);
}

__device__ __forceinline__ void wg_mma(uint32_t d, uint64_t a, uint64_t b, uint32_t idesc, uint32_t accum)
{
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}\n" ::"r"(d),
        "l"(a), "l"(b), "r"(idesc), "r"(accum)
        : "memory");
}

template <bool RAG>
__global__ void __launch_bounds__(TTHREADS)
k_wgrad_tc(const __grid_constant__ CUtensorMap zmap, const __grid_constant__ CUtensorMap xmap,
           const __grid_constant__ CUtensorMap emap, int H, int W, int Cin, int Cout, int ntx, int nty, int ntiles, int per,
           int vec, float *__restrict__ ws)
{
    constexpr int WST = WgLayout<RAG>::ST, WSTAGE = WgLayout<RAG>::STAGE;
    extern __shared__ unsigned char tc_raw[];
    unsigned char *sm = tc_raw + ((1024u - (smem_u32(tc_raw) & 1023u)) & 1023u);
    uint64_t *full = reinterpret_cast<uint64_t *>(sm);  // a stage's copies have landed
    uint64_t *bars = full + WST;                        // the MMAs that read it are complete
    uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(bars + WST);
    unsigned char *stages = sm + 1024;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int c0 = blockIdx.x * 32, co0 = blockIdx.y * TBM;
    const int t0 = blockIdx.z * per, nt = min(per, ntiles - t0);  // at least one tile
    const int atoms = min(4, (Cout - co0 + 31) / 32);
    const long long limit = g_nn_wait_limit;

    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)),
                     "r"(WCOLS)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    if (tid == 0) {
        for (int k = 0; k < WST; ++k) {
            nn_mbar_init(&full[k], 1);
            nn_mbar_init(&bars[k], 1);
        }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    }
    if (tid == 32) {
        asm volatile("prefetch.tensormap [%0];" ::"l"(&zmap) : "memory");
        asm volatile("prefetch.tensormap [%0];" ::"l"(&xmap) : "memory");
    }
    if (RAG && tid >= 64 && tid < 64 + WZERO / 16) {
        *reinterpret_cast<uint4 *>(sm + WgLayout<RAG>::ZERO + (tid - 64) * 16) = make_uint4(0, 0, 0, 0);
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = *tmem_slot;
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");  // after the allocation, as in k_conv3x3_tc
    asm volatile("griddepcontrol.wait;" ::: "memory");

    bool fail = false;
    int k = 0;  // tiles this thread has issued
    if (tid == 32) {  // the copies
        for (; k < nt; ++k) {
            const int st = k % WST, t = t0 + k;
            if (k >= WST && !nn_mbar_wait(&bars[st], uint32_t((k / WST - 1) & 1), limit)) {
                fail = true;
                break;
            }
            unsigned char *base = stages + st * WSTAGE;
            const int x0 = (t % ntx) * TTW, y0 = ((t / ntx) % nty) * TTH, b = t / (ntx * nty);
            const bool edge = RAG && x0 + TTW > W;
            nn_expect(&full[st], uint32_t(atoms * WA_ATOM + (edge ? 2 : 1) * WX_TX));
            for (int a = 0; a < atoms; ++a) nn_tma4(base + a * WA_ATOM, &zmap, &full[st], co0 + a * 32, x0, y0, b);
            nn_tma4(base + WA, &xmap, &full[st], c0, x0 - 1, y0 - 1, b);
            if (edge) nn_tma4(base + WA + WX, &emap, &full[st], c0, W > 1 ? x0 - 1 : 1, y0 - 1, b);
        }
    } else if (tid == 0) {  // the MMAs
        for (; k < nt; ++k) {
            if (!nn_mbar_wait(&full[k % WST], uint32_t((k / WST) & 1), limit)) {
                fail = true;
                break;
            }
            tc_fence_after();
            const uint32_t base = smem_u32(stages + (k % WST) * WSTAGE);
            // A: the next 32 channels an atom further, the next 8 pixels a tile row; B: a pixel, a row with its border
            const uint64_t da0 = wg_desc(base, WA_ATOM, 8 * 64), db0 = wg_desc(base + WA, 64, THW * 64);
            const int rows = min(TTH, H - ((t0 + k) / ntx) % nty * TTH), steps = (rows + 1) / 2;  // past them: zeros
            const bool edge = RAG && ((t0 + k) % ntx) * TTW + TTW > W;
            // the second row of a step from zeros: the K stride of a start address leads there
            const uint32_t zero = smem_u32(sm + WgLayout<RAG>::ZERO);
            auto to_zero = [&](uint64_t d) -> uint64_t {
                const uint64_t stride = (zero >> 4) - (uint32_t)(d & 0x3FFFu);
                return (d & ~((uint64_t)0x3FFFu << 32)) | (stride << 32);
            };
#pragma unroll 2
            for (int r = 0; r < steps; ++r) {
                const uint32_t accum = k > 0 || r > 0;
                const uint64_t da = da0 + (uint64_t)(r * (2 * 8 * 64 / 16));
                const bool half = RAG && 2 * r + 1 == rows;
#pragma unroll
                for (int dy = 0; dy < 3; ++dy) {
                    const uint64_t db = db0 + (uint64_t)((2 * r + dy) * (THW * 64 / 16));
                    const bool z = half && dy == 0;
                    if (!edge) {
                        wg_mma(tmem + dy * 96, da, z ? to_zero(db) : db, wg_idesc(96), accum);
                    } else {
                        const uint64_t dl = db + WX / 16, dc = db + 64 / 16;
                        wg_mma(tmem + dy * 96, da, z ? to_zero(dl) : dl, wg_idesc(32), accum);
                        wg_mma(tmem + dy * 96 + 32, da, z ? to_zero(dc) : dc, wg_idesc(64), accum);
                    }
                }
            }
            asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(
                             smem_u32(&bars[k % WST]))
                         : "memory");
        }
    }
    __syncwarp();
    // every MMA of this block is complete once the commit of the last tile arrives
    const bool done = nn_mbar_wait(&bars[(nt - 1) % WST], uint32_t(((nt - 1) / WST) & 1), limit);
    const bool bad = __syncthreads_or(fail || !done);
    tc_fence_after();
    if (bad) nn_drain(tid, full, bars, WST, k, k);
    {
        // a lane one output channel; two warpgroups split the 18 slices of 16 columns
        const int co = co0 + (warp & 3) * 32 + lane;
        float *o = ws + ((int64_t)blockIdx.z * Cout + co) * 9 * Cin + c0;
#pragma unroll 1
        for (int sl = warp >> 2; sl < 18; sl += 2) {
            uint32_t r[16];
            tmem_ld16(tmem + ((uint32_t)((warp & 3) * 32) << 16) + (uint32_t)(sl * 16), r);
            if (co >= Cout) continue;
            float z[16];
#pragma unroll
            for (int j = 0; j < 16; ++j) z[j] = __uint_as_float(r[j]);
            if (bad)
#pragma unroll
                for (int j = 0; j < 16; ++j) z[j] = NAN;
            float *q = o + (int64_t)(sl >> 1) * Cin + (sl & 1) * 16;
            if (vec) {
                st_v8(q, z);
                st_v8(q + 8, z + 8);
            } else {
#pragma unroll
                for (int j = 0; j < 16; ++j) q[j] = z[j];
            }
        }
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 0)
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(WCOLS) : "memory");
}

struct WgradPlan {
    int ntx, nty, S, per;
};

// The tiles' split over blocks: one block per SM, what its tensor memory lets run
// (us, 148 blocks / 74: 32 -> 32 channels at 128 x 128, batch 16, 20.9 / 34.8; 384 -> 128 at
// 32 x 32 21.5 / 31.9).  A share's length is also the chain its FP32 sums go through.
WgradPlan wgrad_plan(int B, int H, int W, int Cin, int Cout)
{
    WgradPlan p;
    p.ntx = (W + TTW - 1) / TTW;
    p.nty = (H + TTH - 1) / TTH;
    const int64_t tiles = (int64_t)B * p.ntx * p.nty;
    const int64_t bps = (int64_t)((Cin + 31) / 32) * ((Cout + TBM - 1) / TBM);
    int64_t S = bps >= 148 ? 1 : 148 / bps;
    if (S > tiles) S = tiles;
    p.per = int((tiles + S - 1) / S);
    p.S = int((tiles + p.per - 1) / p.per);
    return p;
}

// an image tensor (H x W pixels in memory, the first Hv x Wv of them seen) as (channel, x, y, image): boxes of 32
// channels of w x h pixels, zero outside
bool pixel_map(const void *p, int C, int64_t stride, int B, int Hv, int Wv, int H, int W, int w, int h, CUtensorMap *m)
{
    typedef CUresult (*Encode)(CUtensorMap *, CUtensorMapDataType, cuuint32_t, void *, const cuuint64_t *,
                               const cuuint64_t *, const cuuint32_t *, const cuuint32_t *, CUtensorMapInterleave,
                               CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
    const Encode enc = (Encode)lbm::tensor_map_encoder();
    const cuuint64_t row = (cuuint64_t)stride * 2;
    const cuuint64_t dims[4] = {(cuuint64_t)C, (cuuint64_t)Wv, (cuuint64_t)Hv, (cuuint64_t)B};
    const cuuint64_t str[3] = {row, row * W, row * W * H};
    const cuuint32_t box[4] = {32, (cuuint32_t)w, (cuuint32_t)h, 1}, one[4] = {1, 1, 1, 1};
    return enc && enc(m, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 4, (void *)p, dims, str, box, one,
                      CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_64B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
                      CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

template <bool RAG>
bool launch_wgrad_tc(const bf16 *dz, const bf16 *x, int64_t xs, int xo, int B, int H, int W, int Cin, int Cout,
                     const WgradPlan &pl, float *part, cudaStream_t s)
{
    CUtensorMap zm, xm, em;
    if (!pixel_map(dz, Cout, Cout, B, H, W, H, W, TTW, TTH, &zm) ||
        !pixel_map(x + xo, Cin, xs, B, H, W, H, W, THW, TTH + 2, &xm))
        return false;
    if (!RAG) em = xm;
    else if (!pixel_map(x + xo, Cin, xs, B, H, W > 1 ? W - 1 : 1, H, W, THW, TTH + 2, &em)) return false;
    constexpr int smem = WgLayout<RAG>::SMEM;
    cudaFuncSetAttribute(k_wgrad_tc<RAG>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    const dim3 grid(unsigned(Cin / 32), unsigned((Cout + TBM - 1) / TBM), unsigned(pl.S));
    go(k_wgrad_tc<RAG>, grid, TTHREADS, smem, s, zm, xm, em, H, W, Cin, Cout, pl.ntx, pl.nty, B * pl.ntx * pl.nty, pl.per,
       int(((uintptr_t)part & 31u) == 0), part);
    return true;
}

int g_path = 0;            // lbm_nn_set_tensor_path: 0 the faster kernel for the tensors at hand, 1 tcgen05

}  // namespace

#define NN_REQUIRE(cond, ...)                                         \
    do {                                                              \
        if (!(cond)) return lbm::set_error(LBM_ERR_PARAM, __VA_ARGS__); \
    } while (0)

extern "C" int lbm_nn_conv3x3(const void *x, int64_t xs, int32_t xo, const void *w, const float *bias, int32_t B,
                              int32_t H, int32_t W, int32_t Cin, int32_t Cout, float *of, int64_t os, int32_t oo,
                              int32_t accumulate, void *oa, int64_t as, int32_t ao, int32_t act, void *stream)
{
    NN_REQUIRE(x && w, "lbm_nn_conv3x3: x and w are required");
    NN_REQUIRE(of || oa, "lbm_nn_conv3x3: no output");
    NN_REQUIRE(B > 0 && H > 0 && W > 0 && Cout > 0, "lbm_nn_conv3x3: empty shape");
    NN_REQUIRE(Cin > 0 && Cin % CBK == 0, "lbm_nn_conv3x3: Cin must be a positive multiple of 32");
    NN_REQUIRE(xs % 8 == 0 && xo % 8 == 0 && xo >= 0 && xo + Cin <= xs, "lbm_nn_conv3x3: bad input channel stride/offset");
    NN_REQUIRE(aligned16(x) && aligned16(w), "lbm_nn_conv3x3: x and w must be 16-byte aligned");
    NN_REQUIRE(!of || (oo >= 0 && oo + Cout <= os), "lbm_nn_conv3x3: bad FP32 output stride/offset");
    NN_REQUIRE(!oa || (ao >= 0 && ao + Cout <= as), "lbm_nn_conv3x3: bad bf16 output stride/offset");
    NN_REQUIRE(!accumulate || (!bias && !oa), "lbm_nn_conv3x3: accumulate takes no bias and no bf16 output");
    NN_REQUIRE(act == 0 || act == 1, "lbm_nn_conv3x3: act must be 0 or 1");
    ConvArgs a{(const bf16 *)x, xs, xo, (const bf16 *)w, bias, B, H, W, Cin, Cout, of, os, oo, accumulate,
               (bf16 *)oa, as, ao, act};
    const int64_t M = (int64_t)B * H * W;
    cudaStream_t s = (cudaStream_t)stream;
    // The tcgen05 kernel is the faster on the network's layers and wherever its blocks are some thousand at most.
    // mma.sync takes pixels in a row, across images, and wins where more blocks than that would mostly hold padding
    // (us, tcgen05 / mma.sync: 2000 images of 2 x 2, 64 channels, 31.8 / 19.4; of 1 x 1, 256, 268 / 48; 1000 of 3 x 3, 128,
    // 7 % full, 46.6 / 30.8; but 1000 of 5 x 5, 32, a fifth full, 11.6 / 11.9; 256 of 2 x 2, 256, 1024 blocks, 40.8 / 52.3;
    // 256 of 17 x 3, 64, 12.0 / 19.6).
    const int64_t tiles = tc_tiles(a);
    if (g_path == 1 || 8 * M >= tiles * TTW * TTH || tiles * ((Cout + 63) / 64) <= 1024) {
        if (!conv_tc(a, s)) return lbm::set_error(LBM_ERR_CUDA, "lbm_nn_conv3x3: no tensor maps on this device");
        return launched("lbm_nn_conv3x3 (tcgen05)");
    }
    // ordinary launches: set up while another grid runs, a grid below one wave would share few SMs (128 blocks: 106 us
    // as programmatic dependents of one another, 55 so)
    if (Cout <= 32) {
        dim3 grid(unsigned((M + CBM - 1) / CBM), unsigned((Cout + 31) / 32));
        k_conv3x3<32><<<grid, kThreads, 0, s>>>(a);
    } else {
        dim3 grid(unsigned((M + CBM - 1) / CBM), unsigned((Cout + 63) / 64));
        k_conv3x3<64><<<grid, kThreads, 0, s>>>(a);
    }
    return launched("lbm_nn_conv3x3");
}

extern "C" int lbm_nn_flip_weights(const void *w, void *wt, int32_t Cout, int32_t Cin, void *stream)
{
    NN_REQUIRE(w && wt && Cout > 0 && Cin > 0, "lbm_nn_flip_weights: bad arguments");
    const int64_t n = (int64_t)Cout * 9 * Cin;
    go(k_flip, blocks_for(n), kThreads, 0, (cudaStream_t)stream, (const bf16 *)w, (bf16 *)wt, Cout, Cin);
    return launched("lbm_nn_flip_weights");
}

extern "C" int64_t lbm_nn_wgrad_workspace(int32_t B, int32_t H, int32_t W, int32_t Cin, int32_t Cout)
{
    if (B <= 0 || H <= 0 || W <= 0 || Cin <= 0 || Cout <= 0) return 0;
    const WgradPlan pl = wgrad_plan(B, H, W, Cin, Cout);
    return (int64_t)pl.S * Cout * 9 * Cin;
}

extern "C" int lbm_nn_conv3x3_wgrad(const void *dz, const void *x, int64_t xs, int32_t xo, int32_t B, int32_t H,
                                    int32_t W, int32_t Cin, int32_t Cout, float *ws, int64_t ws_elems, float *dw,
                                    void *stream)
{
    NN_REQUIRE(dz && x && ws && dw, "lbm_nn_conv3x3_wgrad: NULL pointer");
    NN_REQUIRE(B > 0 && H > 0 && W > 0, "lbm_nn_conv3x3_wgrad: empty shape");
    NN_REQUIRE(Cin > 0 && Cin % 32 == 0, "lbm_nn_conv3x3_wgrad: Cin must be a positive multiple of 32");
    NN_REQUIRE(Cout > 0 && Cout % 8 == 0, "lbm_nn_conv3x3_wgrad: Cout must be a positive multiple of 8");
    NN_REQUIRE(xs % 8 == 0 && xo % 8 == 0 && xo >= 0 && xo + Cin <= xs, "lbm_nn_conv3x3_wgrad: bad channel stride/offset");
    NN_REQUIRE(aligned16(dz) && aligned16(x), "lbm_nn_conv3x3_wgrad: dz and x must be 16-byte aligned");
    const WgradPlan pl = wgrad_plan(B, H, W, Cin, Cout);
    const int64_t n = (int64_t)Cout * 9 * Cin;
    NN_REQUIRE(ws_elems >= (int64_t)pl.S * n, "lbm_nn_conv3x3_wgrad: workspace too small (%lld < %lld)",
               (long long)ws_elems, (long long)pl.S * n);
    cudaStream_t s = (cudaStream_t)stream;
    float *part = pl.S == 1 ? dw : ws;  // one share is the sum
    const bool rag = W % TTW != 0 || H % 2 != 0;
    if (!(rag ? launch_wgrad_tc<true> : launch_wgrad_tc<false>)((const bf16 *)dz, (const bf16 *)x, xs, xo, B, H, W, Cin,
                                                                Cout, pl, part, s))
        return lbm::set_error(LBM_ERR_CUDA, "lbm_nn_conv3x3_wgrad: no tensor maps on this device");
    if (pl.S > 1) sum_splits(ws, pl.S, n, dw, s);
    return launched("lbm_nn_conv3x3_wgrad", pl.S > 1 ? 2 : 1);
}

extern "C" int64_t lbm_nn_colsum_workspace(int64_t P, int32_t C)
{
    if (P <= 0 || C <= 0) return 0;
    return ((P + col_rows(P) - 1) / col_rows(P)) * C;
}

// counts the 32-bit index arithmetic of the vector kernels covers
static bool small(int64_t n) { return n < ((int64_t)1 << 32) - kThreads; }

extern "C" int lbm_nn_colsum(const void *a, int64_t P, int32_t C, float *ws, float *out, void *stream)
{
    NN_REQUIRE(a && ws && out && P > 0 && C > 0, "lbm_nn_colsum: bad arguments");
    const int64_t S = (P + col_rows(P) - 1) / col_rows(P);
    cudaStream_t s = (cudaStream_t)stream;
    if (C % 8 == 0 && aligned16(a))
        go(k_colsum8, unsigned(S), kThreads, 0, s, (const bf16 *)a, P, C, ws);
    else
        go(k_colsum, unsigned(S), kThreads, 0, s, (const bf16 *)a, P, C, ws);
    sum_splits(ws, int(S), C, out, s);
    return launched("lbm_nn_colsum", 2);
}

static bool silu_vec(const float *da, int64_t das, int32_t dao, const float *z, int32_t C, const void *dz)
{
    return C % 8 == 0 && das % 4 == 0 && dao % 4 == 0 && aligned16(da) && aligned16(z) && aligned16(dz);
}

extern "C" int lbm_nn_silu_backward(const float *da, int64_t das, int32_t dao, const float *z, int64_t P, int32_t C,
                                    void *dz, void *stream)
{
    NN_REQUIRE(da && z && dz && P > 0 && C > 0 && dao >= 0 && dao + C <= das, "lbm_nn_silu_backward: bad arguments");
    cudaStream_t s = (cudaStream_t)stream;
    if (silu_vec(da, das, dao, z, C, dz))
        go(k_silu_bwd8, unsigned((P + col_rows(P) - 1) / col_rows(P)), kThreads, 0, s, da, das, dao, z, P, C, (bf16 *)dz,
                                                                                 nullptr);
    else
        go(k_silu_bwd, blocks_for(P * C), kThreads, 0, s, da, das, dao, z, P, C, (bf16 *)dz);
    return launched("lbm_nn_silu_backward");
}

extern "C" int lbm_nn_silu_backward_bias(const float *da, int64_t das, int32_t dao, const float *z, int64_t P,
                                         int32_t C, void *dz, float *ws, float *db, void *stream)
{
    NN_REQUIRE(da && z && dz && ws && db && P > 0 && C > 0 && dao >= 0 && dao + C <= das,
               "lbm_nn_silu_backward_bias: bad arguments");
    if (!silu_vec(da, das, dao, z, C, dz)) {
        int st = lbm_nn_silu_backward(da, das, dao, z, P, C, dz, stream);
        return st ? st : lbm_nn_colsum(dz, P, C, ws, db, stream);
    }
    const int64_t S = (P + col_rows(P) - 1) / col_rows(P);
    cudaStream_t s = (cudaStream_t)stream;
    go(k_silu_bwd8, unsigned(S), kThreads, 0, s, da, das, dao, z, P, C, (bf16 *)dz, ws);
    sum_splits(ws, int(S), C, db, s);
    return launched("lbm_nn_silu_backward_bias", 2);
}

extern "C" int lbm_nn_pool2(const void *x, int64_t xs, int32_t xo, int32_t B, int32_t H, int32_t W, int32_t C,
                            void *y, int64_t ys, int32_t yo, void *stream)
{
    NN_REQUIRE(x && y && B > 0 && H > 1 && W > 1 && H % 2 == 0 && W % 2 == 0 && C > 0,
               "lbm_nn_pool2: bad shape (H, W even)");
    NN_REQUIRE(xo >= 0 && xo + C <= xs && yo >= 0 && yo + C <= ys, "lbm_nn_pool2: bad channel stride/offset");
    const int64_t n = (int64_t)B * (H / 2) * (W / 2) * C;
    cudaStream_t s = (cudaStream_t)stream;
    if ((C | xs | xo | ys | yo) % 8 == 0 && aligned16(x) && aligned16(y) && small(n / 8))
        go(k_pool2_v, blocks_for(n / 8), kThreads, 0, s, (const bf16 *)x, xs, xo, B, H, W, C, (bf16 *)y, ys, yo);
    else
        go(k_pool2, blocks_for(n), kThreads, 0, s, (const bf16 *)x, xs, xo, B, H, W, C, (bf16 *)y, ys, yo);
    return launched("lbm_nn_pool2");
}

extern "C" int lbm_nn_pool2_backward(const float *dy, int64_t dys, int32_t dyo, int32_t B, int32_t H, int32_t W,
                                     int32_t C, float *dx, int64_t dxs, int32_t dxo, void *stream)
{
    NN_REQUIRE(dy && dx && B > 0 && H > 1 && W > 1 && H % 2 == 0 && W % 2 == 0 && C > 0,
               "lbm_nn_pool2_backward: bad shape");
    NN_REQUIRE(dyo >= 0 && dyo + C <= dys && dxo >= 0 && dxo + C <= dxs, "lbm_nn_pool2_backward: bad stride/offset");
    const int64_t n = (int64_t)B * H * W * C;
    cudaStream_t s = (cudaStream_t)stream;
    if ((C | dys | dyo | dxs | dxo) % 4 == 0 && aligned16(dy) && aligned16(dx) && small(n / 16))
        go(k_pool2_bwd_v, blocks_for(n / 16), kThreads, 0, s, dy, dys, dyo, B, H, W, C, dx, dxs, dxo);
    else
        go(k_pool2_bwd, blocks_for(n), kThreads, 0, s, dy, dys, dyo, B, H, W, C, dx, dxs, dxo);
    return launched("lbm_nn_pool2_backward");
}

extern "C" int lbm_nn_up2(const void *x, int64_t xs, int32_t xo, int32_t B, int32_t h, int32_t w, int32_t C, void *y,
                          int64_t ys, int32_t yo, void *stream)
{
    NN_REQUIRE(x && y && B > 0 && h > 0 && w > 0 && C > 0, "lbm_nn_up2: bad shape");
    NN_REQUIRE(xo >= 0 && xo + C <= xs && yo >= 0 && yo + C <= ys, "lbm_nn_up2: bad channel stride/offset");
    const int64_t n = (int64_t)B * 4 * h * w * C;
    cudaStream_t s = (cudaStream_t)stream;
    if ((C | xs | xo | ys | yo) % 8 == 0 && aligned16(x) && aligned16(y) && small(n / 32))
        go(k_up2_v, blocks_for(n / 32), kThreads, 0, s, (const bf16 *)x, xs, xo, B, h, w, C, (bf16 *)y, ys, yo);
    else
        go(k_up2, blocks_for(n), kThreads, 0, s, (const bf16 *)x, xs, xo, B, h, w, C, (bf16 *)y, ys, yo);
    return launched("lbm_nn_up2");
}

extern "C" int lbm_nn_up2_backward(const float *dy, int64_t dys, int32_t dyo, int32_t B, int32_t h, int32_t w,
                                   int32_t C, float *dx, int64_t dxs, int32_t dxo, int32_t accumulate, void *stream)
{
    NN_REQUIRE(dy && dx && B > 0 && h > 0 && w > 0 && C > 0, "lbm_nn_up2_backward: bad shape");
    NN_REQUIRE(dyo >= 0 && dyo + C <= dys && dxo >= 0 && dxo + C <= dxs, "lbm_nn_up2_backward: bad stride/offset");
    const int64_t n = (int64_t)B * h * w * C;
    cudaStream_t s = (cudaStream_t)stream;
    if ((C | dys | dyo | dxs | dxo) % 4 == 0 && aligned16(dy) && aligned16(dx) && small(n / 4))
        go(k_up2_bwd_v, blocks_for(n / 4), kThreads, 0, s, dy, dys, dyo, B, h, w, C, dx, dxs, dxo, accumulate);
    else
        go(k_up2_bwd, blocks_for(n), kThreads, 0, s, dy, dys, dyo, B, h, w, C, dx, dxs, dxo, accumulate);
    return launched("lbm_nn_up2_backward");
}

extern "C" int lbm_nn_head(const void *a, int64_t as, int32_t ao, const void *wh, const float *bh, int64_t P, int32_t C,
                           int32_t J, float *y, void *stream)
{
    NN_REQUIRE(a && wh && y && P > 0 && C > 0 && J > 0 && J <= kMaxJ, "lbm_nn_head: bad arguments (J <= 8)");
    NN_REQUIRE(ao >= 0 && ao + C <= as, "lbm_nn_head: bad channel stride/offset");
    cudaStream_t s = (cudaStream_t)stream;
    if (J == 3 && (C | as | ao) % 8 == 0 && aligned16(a))
        go(k_head3_v, blocks_for(P), kThreads, 0, s, (const bf16 *)a, as, ao, (const bf16 *)wh, bh, P, C, y);
    else
        go(k_head, blocks_for(P), kThreads, 0, s, (const bf16 *)a, as, ao, (const bf16 *)wh, bh, P, C, J, y);
    return launched("lbm_nn_head");
}

extern "C" int64_t lbm_nn_head_workspace(int64_t P, int32_t C, int32_t J)
{
    if (P <= 0 || C <= 0 || J <= 0) return 0;
    // per-split partials, then one row for their sums
    return ((P + kHeadRows - 1) / kHeadRows + 1) * ((int64_t)J * C + J);
}

extern "C" int lbm_nn_head_backward(const float *dy, const void *a, int64_t as, int32_t ao, const void *wh, int64_t P,
                                    int32_t C, int32_t J, float *da, int64_t das, int32_t dao, float *ws,
                                    int64_t ws_elems, float *dwh, float *dbh, void *stream)
{
    NN_REQUIRE(dy && a && wh && da && ws && dwh && dbh && P > 0 && C > 0 && J > 0 && J <= kMaxJ,
               "lbm_nn_head_backward: bad arguments");
    NN_REQUIRE(ao >= 0 && ao + C <= as && dao >= 0 && dao + C <= das, "lbm_nn_head_backward: bad stride/offset");
    const int64_t S = (P + kHeadRows - 1) / kHeadRows;
    const int items = J * C + J;
    NN_REQUIRE(ws_elems >= (S + 1) * items, "lbm_nn_head_backward: workspace too small");
    cudaStream_t s = (cudaStream_t)stream;
    if (J == 3 && (C | das | dao) % 4 == 0 && aligned16(da))
        go(k_head3_bwd_da_v, blocks_for(P * C / 4), kThreads, 0, s, dy, (const bf16 *)wh, P, C, da, das, dao);
    else
        go(k_head_bwd_da, blocks_for(P * C), kThreads, 0, s, dy, (const bf16 *)wh, P, C, J, da, das, dao);
    if (J == 3 && (C | as | ao) % 8 == 0 && C <= 256 && aligned16(a))
        go(k_head3_bwd_w_v, unsigned(S), kThreads, 0, s, dy, (const bf16 *)a, as, ao, P, C, ws);
    else
        go(k_head_bwd_w, unsigned(S), kThreads, 0, s, dy, (const bf16 *)a, as, ao, P, C, J, ws);
    // each split's partials hold dwh (J*C) then dbh (J); their ordered sums go after them
    sum_splits(ws, int(S), items, ws + S * items, s);
    int st = launched("lbm_nn_head_backward", 3);
    if (st) return st;
    cudaError_t e = cudaMemcpyAsync(dwh, ws + S * items, sizeof(float) * J * C, cudaMemcpyDeviceToDevice, s);
    if (e == cudaSuccess)
        e = cudaMemcpyAsync(dbh, ws + S * items + (int64_t)J * C, sizeof(float) * J, cudaMemcpyDeviceToDevice, s);
    if (e != cudaSuccess) return lbm::set_error(LBM_ERR_CUDA, "lbm_nn_head_backward: %s", cudaGetErrorString(e));
    return LBM_OK;
}

extern "C" int64_t lbm_nn_mse_workspace(int64_t P, int32_t J)
{
    (void)P;
    (void)J;
    return kMseBlocks;
}

extern "C" int lbm_nn_mse(const float *y, const float *t, const float *cw, int64_t P, int32_t J, float *dy, float *ws,
                          int64_t ws_elems, float *loss, void *stream)
{
    NN_REQUIRE(y && t && dy && ws && loss && P > 0 && J > 0, "lbm_nn_mse: bad arguments");
    NN_REQUIRE(ws_elems >= kMseBlocks, "lbm_nn_mse: workspace too small");
    cudaStream_t s = (cudaStream_t)stream;
    go(k_mse, kMseBlocks, kThreads, 0, s, y, t, cw, P, J, dy, ws);
    go(k_mse_final, 1, 32, 0, s, ws, kMseBlocks, P * J, loss);
    return launched("lbm_nn_mse", 2);
}

extern "C" int lbm_nn_adam(float *p, void *pb, const float *g, float *m, float *v, int64_t n, float lr, float b1,
                           float b2, float eps, float c1, float c2, float wd, void *stream)
{
    NN_REQUIRE(p && g && m && v && n > 0, "lbm_nn_adam: bad arguments");
    NN_REQUIRE(c1 > 0.0f && c2 > 0.0f, "lbm_nn_adam: bias corrections must be > 0");
    go(k_adam, blocks_for(n), kThreads, 0, (cudaStream_t)stream, p, (bf16 *)pb, g, m, v, n, lr, b1, b2, eps, c1, c2, wd);
    return launched("lbm_nn_adam");
}

extern "C" int lbm_nn_to_bf16(const float *x, void *y, int64_t n, void *stream)
{
    NN_REQUIRE(x && y && n > 0, "lbm_nn_to_bf16: bad arguments");
    go(k_to_bf16, blocks_for(n), kThreads, 0, (cudaStream_t)stream, x, (bf16 *)y, n);
    return launched("lbm_nn_to_bf16");
}

extern "C" int lbm_nn_set_tensor_path(int32_t path)
{
    NN_REQUIRE(path == 0 || path == 1, "lbm_nn_set_tensor_path: path must be 0 (automatic) or 1 (tcgen05)");
    g_path = path;
    return LBM_OK;
}

extern "C" int lbm_nn_get_tensor_path(void) { return g_path; }

extern "C" int lbm_nn_timeouts(int32_t *count, int32_t reset)
{
    NN_REQUIRE(count, "lbm_nn_timeouts: count is NULL");
    int v = 0;
    cudaError_t e = cudaMemcpyFromSymbol(&v, g_nn_timeouts, sizeof v);
    if (e == cudaSuccess && reset) {
        const int zero = 0;
        e = cudaMemcpyToSymbol(g_nn_timeouts, &zero, sizeof zero);
    }
    if (e != cudaSuccess) return lbm::set_error(LBM_ERR_CUDA, "lbm_nn_timeouts: %s", cudaGetErrorString(e));
    *count = v;
    return LBM_OK;
}

extern "C" int lbm_nn_set_wait_limit(int64_t cycles)
{
    NN_REQUIRE(cycles >= 0, "lbm_nn_set_wait_limit: the limit must be >= 0");
    const long long v = cycles > 0 ? cycles : kNnWaitCycles;
    const cudaError_t e = cudaMemcpyToSymbol(g_nn_wait_limit, &v, sizeof v);
    if (e != cudaSuccess) return lbm::set_error(LBM_ERR_CUDA, "lbm_nn_set_wait_limit: %s", cudaGetErrorString(e));
    return LBM_OK;
}

// ---------------------------------------------------------------------------
// the network's passes
// ---------------------------------------------------------------------------
// One call issues the pass's launches: from Python each launch is a foreign call
// of some twenty arguments, 8 us, as much as the kernels take at batch 1.  One
// prediction at 128 x 128: the host's share 175 -> 91 us, the pass 173 -> 156 us
// (with the kernels since: 78 and 112).
#define NN_DO(call)                   \
    do {                              \
        const int st_ = (call);       \
        if (st_ != LBM_OK) return st_; \
    } while (0)

namespace {

// a layer's image size, and its input and output tensors
struct UnetLayer {
    const void *x;
    int xs;
    void *a;
    int as, ao, H;
};

void unet_layers(const lbm_nn_unet &n, UnetLayer l[14])
{
    const int c1 = n.ch[0][1], c2 = n.ch[2][1], c3 = n.ch[4][1], c4 = n.ch[6][1], R = n.R;
    const int k1 = c2 + c1, k2 = c3 + c2, k3 = c4 + c3;  // channels of the concat buffers
    const UnetLayer t[14] = {
        {n.x, n.ch[0][0], n.a[0], c1, 0, R},         {n.a[0], c1, n.cat[0], k1, c2, R},
        {n.p[0], c1, n.a[2], c2, 0, R / 2},          {n.a[2], c2, n.cat[1], k2, c3, R / 2},
        {n.p[1], c2, n.a[4], c3, 0, R / 4},          {n.a[4], c3, n.cat[2], k3, c4, R / 4},
        {n.p[2], c3, n.a[6], c4, 0, R / 8},          {n.a[6], c4, n.a[7], c4, 0, R / 8},
        {n.cat[2], k3, n.a[8], c3, 0, R / 4},        {n.a[8], c3, n.a[9], c3, 0, R / 4},
        {n.cat[1], k2, n.a[10], c2, 0, R / 2},       {n.a[10], c2, n.a[11], c2, 0, R / 2},
        {n.cat[0], k1, n.a[12], c1, 0, R},           {n.a[12], c1, n.a[13], c1, 0, R}};
    for (int k = 0; k < 14; ++k) l[k] = t[k];
}

int unet_check(const lbm_nn_unet *n, const char *what)
{
    NN_REQUIRE(n && n->B > 0 && n->R >= 16 && n->R % 8 == 0 && n->J > 0, "%s: bad arguments", what);
    NN_REQUIRE(n->pb && n->master, "%s: NULL parameters", what);
    return LBM_OK;
}

const char *at16(const void *p, int64_t o) { return (const char *)p + 2 * o; }

}  // namespace

extern "C" int lbm_nn_unet_forward(const lbm_nn_unet *net, void *stream)
{
    NN_DO(unet_check(net, "lbm_nn_unet_forward"));
    const lbm_nn_unet &n = *net;
    const int B = n.B;
    UnetLayer l[14];
    unet_layers(n, l);
    for (int k = 0; k < 14; ++k) {
        const UnetLayer &t = l[k];
        const int ci = n.ch[k][0], co = n.ch[k][1], H = t.H;
        NN_DO(lbm_nn_conv3x3(t.x, t.xs, 0, at16(n.pb, n.off[k][0]), n.master + n.off[k][1], B, H, H, ci, co, n.z[k], co,
                             0, 0, t.a, t.as, t.ao, 1, stream));
        if (k == 1 || k == 3 || k == 5)  // the end of an encoder level
            NN_DO(lbm_nn_pool2(t.a, t.as, t.ao, B, H, H, co, n.p[k / 2], co, 0, stream));
        if (k == 7 || k == 9 || k == 11) {  // up into the next decoder level
            const int d = (11 - k) / 2;
            NN_DO(lbm_nn_up2(t.a, co, 0, B, H, H, co, n.cat[d], l[k + 1].xs, 0, stream));
        }
    }
    return lbm_nn_head(n.a[13], l[13].as, 0, at16(n.pb, n.off[14][0]), n.master + n.off[14][1], (int64_t)B * n.R * n.R,
                       l[13].as, n.J, n.y, stream);
}

extern "C" int lbm_nn_unet_backward(const lbm_nn_unet *net, void *stream)
{
    NN_DO(unet_check(net, "lbm_nn_unet_backward"));
    const lbm_nn_unet &n = *net;
    NN_REQUIRE(n.wt && n.grad && n.dy && n.ws, "lbm_nn_unet_backward: NULL pointer");
    const int B = n.B;
    UnetLayer l[14];
    unet_layers(n, l);
    // every pass of the chain uses the one scratch, the column sums without a size of their own
    int64_t need = lbm_nn_head_workspace((int64_t)B * n.R * n.R, l[13].as, n.J);
    for (int k = 0; k < 14; ++k) {
        const int ci = n.ch[k][0], co = n.ch[k][1], H = l[k].H;
        need = std::max({need, lbm_nn_wgrad_workspace(B, H, H, ci, co), lbm_nn_colsum_workspace((int64_t)B * H * H, co)});
    }
    NN_REQUIRE(n.ws_elems >= need, "lbm_nn_unet_backward: workspace too small (%lld < %lld)", (long long)n.ws_elems,
               (long long)need);
    for (int k = 0; k < 14; ++k)
        NN_DO(lbm_nn_flip_weights(at16(n.pb, n.off[k][0]), (char *)n.wt + 2 * n.off[k][0], n.ch[k][1], n.ch[k][0],
                                  stream));
    NN_DO(lbm_nn_head_backward(n.dy, n.a[13], l[13].as, 0, at16(n.pb, n.off[14][0]), (int64_t)B * n.R * n.R, l[13].as,
                               n.J, n.da[13], l[13].as, 0, n.ws, n.ws_elems, n.grad + n.off[14][0],
                               n.grad + n.off[14][1], stream));
    // where a layer's input gradient goes, per layer: its tensor and channel stride
    float *const dx[14] = {nullptr, n.da[0], n.dp[0], n.da[2], n.dp[1], n.da[4], n.dp[2], n.da[6], n.dcat[2], n.da[8],
                           n.dcat[1], n.da[10], n.dcat[0], n.da[12]};
    for (int k = 13; k >= 0; --k) {
        const UnetLayer &t = l[k];
        const int ci = n.ch[k][0], co = n.ch[k][1], H = t.H;
        const bool skip = k == 1 || k == 3 || k == 5;  // its output is the skip half of a concat buffer
        const float *da = skip ? n.dcat[k / 2] : n.da[k];
        NN_DO(lbm_nn_silu_backward_bias(da, t.as, t.ao, n.z[k], (int64_t)B * H * H, co, n.dz[k], n.ws,
                                        n.grad + n.off[k][1], stream));
        NN_DO(lbm_nn_conv3x3_wgrad(n.dz[k], t.x, t.xs, 0, B, H, H, ci, co, n.ws, n.ws_elems, n.grad + n.off[k][0],
                                   stream));
        if (dx[k])
            NN_DO(lbm_nn_conv3x3(n.dz[k], co, 0, (char *)n.wt + 2 * n.off[k][0], nullptr, B, H, H, co, ci, dx[k], t.xs, 0,
                                 0, nullptr, 0, 0, 0, stream));
        if (k == 12 || k == 10 || k == 8) {  // the upsampled half of the concat buffer
            const int up = n.ch[k - 1][1];
            NN_DO(lbm_nn_up2_backward(dx[k], t.xs, 0, B, H / 2, H / 2, up, n.da[k - 1], up, 0, 0, stream));
        }
        if (k == 6 || k == 4 || k == 2) {  // through the pooling into the skip half
            const int e = k / 2 - 1, c = n.ch[k - 1][1];
            NN_DO(lbm_nn_pool2_backward(n.dp[e], c, 0, B, 2 * H, 2 * H, c, n.dcat[e], l[k - 1].as, l[k - 1].ao, stream));
        }
    }
    return LBM_OK;
}
