// bun_elem.cu -- the U-Net's CUDA-core kernels: the 1-channel input
// convolution and the 1x1x1 output head (too narrow for a tensor-core tile),
// pooling and its gradients, the loss, weight packing for the tensor-core
// convolutions, Adam, and the scalings between the solver's FP64 fields and
// the network's FP32 input/output.  Most are a pass over memory; the input layer
// is bound by its multiply-adds (8 % of a forward pass at 256^3).  Reductions
// write one partial per block and are added in a fixed order.

#include "bun_api_internal.h"

#include <cstdint>
#include <initializer_list>

namespace bun {

namespace {

constexpr int kBlock = 256;

// (a grid has at most 2^30 voxels: 32-bit divisions)
__device__ __forceinline__ void decode(long v, int n1, int n2, int& i, int& j, int& k) {
    const unsigned u = (unsigned)v, q = u / (unsigned)n2;
    k = (int)(u - q * (unsigned)n2);
    i = (int)(q / (unsigned)n1);
    j = (int)(q - (unsigned)i * (unsigned)n1);
}

// 8 channels: one 16-byte vector
__device__ __forceinline__ void ld8(const bf16* p, float v[8]) {
    const uint4 a = *reinterpret_cast<const uint4*>(p);
    const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&a);
#pragma unroll
    for (int q = 0; q < 4; ++q) {
        const float2 f = __bfloat1622float2(h[q]);
        v[2 * q] = f.x;
        v[2 * q + 1] = f.y;
    }
}
__device__ __forceinline__ void st8(bf16* p, const float v[8]) {
    uint4 a;
    __nv_bfloat162* h = reinterpret_cast<__nv_bfloat162*>(&a);
#pragma unroll
    for (int q = 0; q < 4; ++q) h[q] = __floats2bfloat162_rn(v[2 * q], v[2 * q + 1]);
    *reinterpret_cast<uint4*>(p) = a;
}
// channels in whole vectors, arrays on 16 bytes
inline bool vec8(std::initializer_list<int> channels, std::initializer_list<const void*> arrays) {
    for (int c : channels)
        if (c % 8) return false;
    for (const void* p : arrays)
        if (reinterpret_cast<uintptr_t>(p) & 15u) return false;
    return true;
}

__device__ __forceinline__ float block_sum(float x, float* sh) {
    for (int o = 16; o > 0; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    __syncthreads();
    if (lane == 0) sh[warp] = x;
    __syncthreads();
    x = 0.f;
    if (warp == 0) {
        x = lane < (int)(blockDim.x >> 5) ? sh[lane] : 0.f;
        for (int o = 16; o > 0; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
    }
    return x;
}

// a0[v][c] = relu(b[c] + sum_t w[t][c] x[v + off(t)])   (1 -> 16 channels)
// A block owns kInJ rows x kInK voxels of one plane: it stages the input
// tile with its one-voxel halo (zero outside the grid) in shared memory
// once, so each input value is read from memory about once instead of 27
// times.  A thread forms four voxels (rows tj, tj + kInJ/4, ...), reading
// each tap's weights four channels at a time, so one shared-memory load
// feeds sixteen FMAs.
constexpr int kInK = 64, kInJ = 16;  // kInK * kInJ == 4 * kBlock
constexpr int kInI = 8;              // most planes a CTA
// A CTA walks up to kInI planes of its tile with the input planes in a ring of
// four, the next one's copies under this one's arithmetic, so a plane is fetched
// once and not three times with every load waited for: 256^3 543 -> 365 us. Bound
// by the multiply-adds (432 a voxel, two channels an instruction: 200 us of issue)
// and the weights' shared loads between them.
__global__ void __launch_bounds__(kBlock, 2) k_conv_in(int n0, int n1, int n2, int planes,
                                                       const float* __restrict__ x, const float* __restrict__ w,
                                                       const float* __restrict__ b, bf16* __restrict__ out) {
    constexpr int SK = kInK + 2, PL = (kInJ + 2) * SK, NL = (PL + kBlock - 1) / kBlock;
    __shared__ __align__(16) float sw[27 * 16 + 16];
    __shared__ float sx[4][PL];
    for (int q = threadIdx.x; q < 27 * 16; q += blockDim.x) sw[q] = w[q];
    if (threadIdx.x < 16) sw[27 * 16 + threadIdx.x] = b[threadIdx.x];
    const int k0 = blockIdx.x * kInK, j0 = blockIdx.y * kInJ;
    const int is = blockIdx.z * planes, ie = min(is + planes, n0);
    const long plane = (long)n1 * n2;
    // this thread's values of a plane: offset in the plane, -1 outside the grid
    long off[NL];
#pragma unroll
    for (int m = 0; m < NL; ++m) {
        const int r = threadIdx.x + m * kBlock, dj = r / SK, dk = r - dj * SK;
        const int jj = j0 + dj - 1, kk = k0 + dk - 1;
        off[m] = r < PL && jj >= 0 && jj < n1 && kk >= 0 && kk < n2 ? (long)jj * n2 + kk : -1;
    }
    auto fetch = [&](int ii) {
        const bool in = ii >= 0 && ii < n0;
        const float* xp = x + (in ? ii : 0) * plane;
        const uint32_t d = (uint32_t)__cvta_generic_to_shared(sx[(ii + 4) & 3]) + 4 * threadIdx.x;
#pragma unroll
        for (int m = 0; m < NL; ++m) {
            if (threadIdx.x + m * kBlock >= PL) break;
            const bool v = in && off[m] >= 0;
            asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(d + m * kBlock * 4),
                         "l"(v ? xp + off[m] : x), "r"(v ? 4 : 0)
                         : "memory");
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    fetch(is - 1);
    fetch(is);
    fetch(is + 1);
    constexpr int RJ = kInJ / 4;  // rows between a thread's voxels
    const int tk = threadIdx.x % kInK, tj = threadIdx.x / kInK;
    const int k = k0 + tk;
#pragma unroll 1
    for (int i = is; i < ie; ++i) {
        asm volatile("cp.async.wait_group 0;" ::: "memory");
        __syncthreads();
        if (i + 1 < ie) fetch(i + 2);  // into plane i - 2, which no thread reads any more
        // pairs of channels: one packed instruction per two multiply-adds
        unsigned long long acc2[4][8];
        const unsigned long long* sw2 = reinterpret_cast<const unsigned long long*>(sw);
#pragma unroll
        for (int u = 0; u < 4; ++u)
#pragma unroll
            for (int c = 0; c < 8; ++c) acc2[u][c] = sw2[27 * 8 + c];
#pragma unroll 1
        for (int t3 = 0; t3 < 9; ++t3) {
            const int di = t3 / 3, dj = t3 - 3 * di;
            const float* sp = &sx[(i + di + 3) & 3][(tj + dj) * SK + tk];
#pragma unroll
            for (int dk = 0; dk < 3; ++dk) {
                unsigned long long xv[4];
#pragma unroll
                for (int u = 0; u < 4; ++u) {
                    const float x1 = sp[u * RJ * SK + dk];
                    asm("mov.b64 %0, {%1, %1};" : "=l"(xv[u]) : "f"(x1));
                }
                const ulonglong2* wt = reinterpret_cast<const ulonglong2*>(sw + (t3 * 3 + dk) * 16);
#pragma unroll
                for (int g = 0; g < 4; ++g) {
                    const ulonglong2 wv = wt[g];
#pragma unroll
                    for (int u = 0; u < 4; ++u) {
                        asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(acc2[u][2 * g]) : "l"(wv.x), "l"(xv[u]));
                        asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(acc2[u][2 * g + 1]) : "l"(wv.y), "l"(xv[u]));
                    }
                }
            }
        }
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            const int j = j0 + tj + u * RJ;
            if (j >= n1 || k >= n2) continue;
            uint4 ov[2];
            __nv_bfloat162* o = reinterpret_cast<__nv_bfloat162*>(ov);
#pragma unroll
            for (int q = 0; q < 8; ++q) {
                float lo, hi;
                asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(acc2[u][q]));
                o[q] = __floats2bfloat162_rn(fmaxf(lo, 0.f), fmaxf(hi, 0.f));
            }
            uint4* op = reinterpret_cast<uint4*>(out + (((long)i * n1 + j) * n2 + k) * 16);
            op[0] = ov[0];
            op[1] = ov[1];
        }
    }
}

// partials of dW[t][c] = sum_v x[v+off(t)] dz[v][c] (t < 27) and db[c] =
// sum_v dz[v][c] (t = 27): part[blk][t*16 + c].  Eight lanes hold all taps of two
// channels each and march along k over runs of kInRun voxels with the nine rows'
// three columns in registers, so dz is read once, and x nine values a step: bound
// by the 56 sums a step.  A CTA for every tap, then three taps, read dz 28 and
// ten times: 346 and 206 us at 128^3, now 146.
// A run's sums go to totals in shared memory (two channels a word, a column a
// thread): a chain of FP32 additions is a run's voxels or the thread's runs
// long, not their product, which at 256^3 had 2048 terms and lost to the
// thread-per-voxel kernel's 256 (relative error against 64 bits 8.5e-7, now 3.4e-7;
// that kernel 3.7e-7); the totals cost no time that shows (1134 -> 1123 us).
constexpr int kInRun = 32;
constexpr int kInTotals = 28 * kBlock * (int)sizeof(float2);
__global__ void __launch_bounds__(kBlock, 2) k_conv_in_wgrad(int n0, int n1, int n2, const float* __restrict__ x,
                                                             const bf16* __restrict__ dz, float* __restrict__ part) {
    constexpr int WARPS = kBlock / 32;
    __shared__ float sh[WARPS][28 * 16];
    extern __shared__ float2 total[];  // [28][kBlock]
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, c2 = lane & 7;
    const int nr = (n2 + kInRun - 1) / kInRun;
    const long runs = (long)n0 * n1 * nr, groups = (long)gridDim.x * (kBlock / 8);
    // (zeros the compiler does not see: it would peel the first steps of a run and spill)
    auto zero = [](float& v) { asm volatile("mov.b32 %0, 0;" : "=f"(v)); };
    float acc[28][2];
#pragma unroll
    for (int t = 0; t < 28; ++t) {
        zero(acc[t][0]);
        zero(acc[t][1]);
        total[t * kBlock + threadIdx.x] = make_float2(0.f, 0.f);
    }
#pragma unroll 1
    for (long g = ((long)blockIdx.x * kBlock + threadIdx.x) >> 3; g < runs; g += groups) {
        int i, j, q;
        decode(g, n1, nr, i, j, q);
        const int ks = q * kInRun, ke = min(ks + kInRun, n2);
        const float* row = x + ((long)i * n1 + j) * n2;
        const bf16* dr = dz + (((long)i * n1 + j) * n2) * 16 + 2 * c2;
        bool in[9];  // the nine rows inside the grid
#pragma unroll
        for (int r = 0; r < 9; ++r) {
            const int ii = i + r / 3 - 1, jj = j + r % 3 - 1;
            in[r] = ii >= 0 && ii < n0 && jj >= 0 && jj < n1;
        }
        float xm[9], xc[9], xp[9];
#pragma unroll
        for (int r = 0; r < 9; ++r) {
            const float* p = row + ((long)(r / 3 - 1) * n1 + (r % 3 - 1)) * n2;
            xm[r] = in[r] && ks > 0 ? p[ks - 1] : 0.f;
            xc[r] = in[r] ? p[ks] : 0.f;
        }
#pragma unroll 3
        for (int k = ks; k < ke; ++k) {
#pragma unroll
            for (int r = 0; r < 9; ++r) {
                const float* p = row + ((long)(r / 3 - 1) * n1 + (r % 3 - 1)) * n2;
                xp[r] = in[r] && k + 1 < n2 ? p[k + 1] : 0.f;
            }
            const float2 d = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(dr + (long)k * 16));
#pragma unroll
            for (int r = 0; r < 9; ++r) {
                acc[3 * r][0] += xm[r] * d.x;
                acc[3 * r][1] += xm[r] * d.y;
                acc[3 * r + 1][0] += xc[r] * d.x;
                acc[3 * r + 1][1] += xc[r] * d.y;
                acc[3 * r + 2][0] += xp[r] * d.x;
                acc[3 * r + 2][1] += xp[r] * d.y;
                xm[r] = xc[r];
                xc[r] = xp[r];
            }
            acc[27][0] += d.x;
            acc[27][1] += d.y;
        }
#pragma unroll
        for (int t = 0; t < 28; ++t) {
            float2& s = total[t * kBlock + threadIdx.x];
            s = make_float2(s.x + acc[t][0], s.y + acc[t][1]);
            zero(acc[t][0]);
            zero(acc[t][1]);
        }
    }
    // the warp's four groups, then the warps
#pragma unroll
    for (int t = 0; t < 28; ++t) {
        float2 v = total[t * kBlock + threadIdx.x];
#pragma unroll
        for (int o = 8; o <= 16; o *= 2) {
            v.x += __shfl_xor_sync(0xffffffffu, v.x, o);
            v.y += __shfl_xor_sync(0xffffffffu, v.y, o);
        }
        if (lane < 8) {
            sh[warp][t * 16 + 2 * c2] = v.x;
            sh[warp][t * 16 + 2 * c2 + 1] = v.y;
        }
    }
    __syncthreads();
    for (int q = threadIdx.x; q < 28 * 16; q += kBlock) {
        float v = 0.f;
#pragma unroll
        for (int w = 0; w < WARPS; ++w) v += sh[w][q];
        part[(long)blockIdx.x * (28 * 16) + q] = v;
    }
}

// y[v] = b + sum_c w[c] d[v][c]    (16 -> 1 channel, 1x1x1)
__global__ void __launch_bounds__(kBlock) k_head(long V, const bf16* __restrict__ d, const float* __restrict__ w,
                                                 const float* __restrict__ b, float* __restrict__ y) {
    const long v = (long)blockIdx.x * blockDim.x + threadIdx.x;
    if (v >= V) return;
    const uint4* dp = reinterpret_cast<const uint4*>(d + v * 16);
    uint4 dv[2] = {dp[0], dp[1]};
    const bf16* e = reinterpret_cast<const bf16*>(dv);
    float acc = b[0];
#pragma unroll
    for (int c = 0; c < 16; ++c) acc += w[c] * __bfloat162float(e[c]);
    y[v] = acc;
}

// dz[v][c] = dy[v] w[c] (d[v][c] > 0); partials of dW[c] = sum dy d and db
__global__ void __launch_bounds__(kBlock) k_head_grad(long V, const bf16* __restrict__ d,
                                                      const float* __restrict__ dy, const float* __restrict__ w,
                                                      bf16* __restrict__ dz, float* __restrict__ part) {
    __shared__ float sh[kBlock / 32];
    float acc[17];
#pragma unroll
    for (int c = 0; c < 17; ++c) acc[c] = 0.f;
    for (long v = (long)blockIdx.x * blockDim.x + threadIdx.x; v < V; v += (long)gridDim.x * blockDim.x) {
        const uint4* dp = reinterpret_cast<const uint4*>(d + v * 16);
        uint4 dv[2] = {dp[0], dp[1]};
        const bf16* e = reinterpret_cast<const bf16*>(dv);
        const float g = dy[v];
        uint4 ov[2];
        __nv_bfloat162* o = reinterpret_cast<__nv_bfloat162*>(ov);
#pragma unroll
        for (int q = 0; q < 8; ++q) {
            const float a0 = __bfloat162float(e[2 * q]), a1 = __bfloat162float(e[2 * q + 1]);
            o[q] = __floats2bfloat162_rn(a0 > 0.f ? g * w[2 * q] : 0.f, a1 > 0.f ? g * w[2 * q + 1] : 0.f);
            acc[2 * q] += g * a0;
            acc[2 * q + 1] += g * a1;
        }
        acc[16] += g;
        uint4* op = reinterpret_cast<uint4*>(dz + v * 16);
        op[0] = ov[0];
        op[1] = ov[1];
    }
#pragma unroll
    for (int c = 0; c < 17; ++c) {
        const float s = block_sum(acc[c], sh);
        if (threadIdx.x == 0) part[(long)blockIdx.x * 17 + c] = s;
    }
}

// p[w][c] = mean of the 8 children of coarse voxel w (fine grid n0 x n1 x n2)
__global__ void __launch_bounds__(kBlock) k_pool(int n0, int n1, int n2, int C, const bf16* __restrict__ s,
                                                 bf16* __restrict__ p) {
    const int m0 = n0 / 2, m1 = n1 / 2, m2 = n2 / 2;
    const long total = (long)m0 * m1 * m2 * (C / 2);
    const long q = (long)blockIdx.x * blockDim.x + threadIdx.x;
    if (q >= total) return;
    const int c2 = (int)(q % (C / 2));
    const long w = q / (C / 2);
    int I, J, K;
    decode(w, m1, m2, I, J, K);
    float a0 = 0.f, a1 = 0.f;
#pragma unroll
    for (int o = 0; o < 8; ++o) {
        const long f = ((long)(2 * I + (o >> 2)) * n1 + 2 * J + ((o >> 1) & 1)) * n2 + 2 * K + (o & 1);
        const float2 v = __bfloat1622float2(reinterpret_cast<const __nv_bfloat162*>(s + f * C)[c2]);
        a0 += v.x;
        a1 += v.y;
    }
    reinterpret_cast<__nv_bfloat162*>(p + w * C)[c2] = __floats2bfloat162_rn(0.125f * a0, 0.125f * a1);
}

// the same for 8 channels a thread, as one vector of every child (256^3, 16
// channels: 159 -> 85 us)
__global__ void __launch_bounds__(kBlock) k_pool8(int n0, int n1, int n2, int C, const bf16* __restrict__ s,
                                                  bf16* __restrict__ p) {
    const int m0 = n0 / 2, m1 = n1 / 2, m2 = n2 / 2;
    const unsigned nc = (unsigned)C / 8;
    const long q = (long)blockIdx.x * blockDim.x + threadIdx.x;
    if (q >= (long)m0 * m1 * m2 * nc) return;
    const unsigned w = (unsigned)q / nc, c = 8 * ((unsigned)q - w * nc);
    int I, J, K;
    decode(w, m1, m2, I, J, K);
    float a[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
#pragma unroll
    for (int o = 0; o < 8; ++o) {
        const long f = ((long)(2 * I + (o >> 2)) * n1 + 2 * J + ((o >> 1) & 1)) * n2 + 2 * K + (o & 1);
        float v[8];
        ld8(s + f * C + c, v);
#pragma unroll
        for (int e = 0; e < 8; ++e) a[e] += v[e];
    }
#pragma unroll
    for (int e = 0; e < 8; ++e) a[e] *= 0.125f;
    st8(p + (long)w * C + c, a);
}

// gradient of the upsampled part of a concatenated input: for coarse voxel
// w and channel c < c0, dz[w][c] = (sum over children of dcat[f][c]) *
// (act[w][c] > 0)
__global__ void __launch_bounds__(kBlock) k_unpool_grad(int n0, int n1, int n2, int ccat, int c0,
                                                        const bf16* __restrict__ dcat,
                                                        const bf16* __restrict__ act, bf16* __restrict__ dz) {
    const int m0 = n0 / 2, m1 = n1 / 2, m2 = n2 / 2;
    const long total = (long)m0 * m1 * m2 * c0;
    const long q = (long)blockIdx.x * blockDim.x + threadIdx.x;
    if (q >= total) return;
    const int c = (int)(q % c0);
    const long w = q / c0;
    int I, J, K;
    decode(w, m1, m2, I, J, K);
    float a = 0.f;
#pragma unroll
    for (int o = 0; o < 8; ++o) {
        const long f = ((long)(2 * I + (o >> 2)) * n1 + 2 * J + ((o >> 1) & 1)) * n2 + 2 * K + (o & 1);
        a += __bfloat162float(dcat[f * ccat + c]);
    }
    dz[w * c0 + c] = __float2bfloat16_rn(__bfloat162float(act[w * c0 + c]) > 0.f ? a : 0.f);
}

__global__ void __launch_bounds__(kBlock) k_unpool_grad8(int n0, int n1, int n2, int ccat, int c0,
                                                         const bf16* __restrict__ dcat,
                                                         const bf16* __restrict__ act, bf16* __restrict__ dz) {
    const int m0 = n0 / 2, m1 = n1 / 2, m2 = n2 / 2;
    const unsigned nc = (unsigned)c0 / 8;
    const long q = (long)blockIdx.x * blockDim.x + threadIdx.x;
    if (q >= (long)m0 * m1 * m2 * nc) return;
    const unsigned w = (unsigned)q / nc, c = 8 * ((unsigned)q - w * nc);
    int I, J, K;
    decode(w, m1, m2, I, J, K);
    float a[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f}, m[8];
#pragma unroll
    for (int o = 0; o < 8; ++o) {
        const long f = ((long)(2 * I + (o >> 2)) * n1 + 2 * J + ((o >> 1) & 1)) * n2 + 2 * K + (o & 1);
        float v[8];
        ld8(dcat + f * ccat + c, v);
#pragma unroll
        for (int e = 0; e < 8; ++e) a[e] += v[e];
    }
    ld8(act + (long)w * c0 + c, m);
#pragma unroll
    for (int e = 0; e < 8; ++e) a[e] = m[e] > 0.f ? a[e] : 0.f;
    st8(dz + (long)w * c0 + c, a);
}

// gradient of a skip tensor s (C channels, fine grid), used both by the
// decoder's concatenation (channels [c0, c0 + C) of dcat) and by the pooling
// that feeds the next encoder level (dp, coarse grid):
//   dz[v][c] = (s[v][c] > 0) * (dcat[v][c0 + c] + dp[parent(v)][c] / 8)
__global__ void __launch_bounds__(kBlock) k_skip_grad(int n0, int n1, int n2, int ccat, int c0, int C,
                                                      const bf16* __restrict__ dcat, const bf16* __restrict__ dp,
                                                      const bf16* __restrict__ s, bf16* __restrict__ dz) {
    const long total = (long)n0 * n1 * n2 * C;
    const long q = (long)blockIdx.x * blockDim.x + threadIdx.x;
    if (q >= total) return;
    const int c = (int)(q % C);
    const long v = q / C;
    int i, j, k;
    decode(v, n1, n2, i, j, k);
    const long w = ((long)(i >> 1) * (n1 >> 1) + (j >> 1)) * (n2 >> 1) + (k >> 1);
    const float g = __bfloat162float(dcat[v * ccat + c0 + c]) + 0.125f * __bfloat162float(dp[w * C + c]);
    dz[v * C + c] = __float2bfloat16_rn(__bfloat162float(s[v * C + c]) > 0.f ? g : 0.f);
}

// (16 channels on 128^3: 192 -> 48 us; one channel a thread, with 64-bit
// divisions for each, before)
__global__ void __launch_bounds__(kBlock) k_skip_grad8(int n0, int n1, int n2, int ccat, int c0, int C,
                                                       const bf16* __restrict__ dcat, const bf16* __restrict__ dp,
                                                       const bf16* __restrict__ s, bf16* __restrict__ dz) {
    const unsigned nc = (unsigned)C / 8;
    const long q = (long)blockIdx.x * blockDim.x + threadIdx.x;
    if (q >= (long)n0 * n1 * n2 * nc) return;
    const long v = q / nc;
    const int c = 8 * (int)(q - v * nc);
    int i, j, k;
    decode(v, n1, n2, i, j, k);
    const long w = ((long)(i >> 1) * (n1 >> 1) + (j >> 1)) * (n2 >> 1) + (k >> 1);
    float a[8], b[8], m[8];
    ld8(dcat + v * ccat + c0 + c, a);
    ld8(dp + w * C + c, b);
    ld8(s + v * C + c, m);
#pragma unroll
    for (int e = 0; e < 8; ++e) a[e] = m[e] > 0.f ? a[e] + 0.125f * b[e] : 0.f;
    st8(dz + v * C + c, a);
}

// dy = 2 (y - t) / n; partials of sum (y - t)^2
__global__ void __launch_bounds__(kBlock) k_mse(long n, const float* __restrict__ y, const float* __restrict__ t,
                                                float* __restrict__ dy, float* __restrict__ part) {
    __shared__ float sh[kBlock / 32];
    float acc = 0.f;
    const float sc = 2.f / (float)n;
    for (long v = (long)blockIdx.x * blockDim.x + threadIdx.x; v < n; v += (long)gridDim.x * blockDim.x) {
        const float e = y[v] - t[v];
        dy[v] = sc * e;
        acc += e * e;
    }
    acc = block_sum(acc, sh);
    if (threadIdx.x == 0) part[blockIdx.x] = acc;
}

// out[q] = scale * sum_p part[p * stride + q], p in fixed order
__global__ void __launch_bounds__(kBlock) k_sum_parts(const float* __restrict__ part, int nparts, long stride,
                                                      long len, float scale, float* __restrict__ out) {
    const long q = (long)blockIdx.x * blockDim.x + threadIdx.x;
    if (q >= len) return;
    float a = 0.f;
    for (int p = 0; p < nparts; ++p) a += part[(long)p * stride + q];
    out[q] = scale * a;
}

// packed weights of one tensor-core convolution.  Forward (transpose = 0):
// GEMM K = cin, N = cout, element (n = co, c = ci) of block (t, g) holds
// W[t][g*kc + c][co].  Data gradient (transpose = 1): K = cout, N = cin,
// element (n = ci, c = co) of block (t, g) holds W[26 - t][ci][g*kc + c].
// Inside a block: element (n/8)*(kc*8) + (c/8)*64 + (n%8)*8 + (c%8).
__global__ void __launch_bounds__(kBlock) k_pack(const float* __restrict__ w, int cin, int cout, int kc,
                                                 int transpose, bf16* __restrict__ out) {
    const int K = transpose ? cout : cin, N = transpose ? cin : cout;
    const long total = 27L * K * N;
    const long q = (long)blockIdx.x * blockDim.x + threadIdx.x;
    if (q >= total) return;
    const long blk = q / ((long)N * kc);
    const int r = (int)(q % ((long)N * kc));
    const int ng = r / (kc * 8);
    const int r2 = r % (kc * 8);
    const int cg = r2 / 64, r3 = r2 % 64;
    const int nr = r3 / 8, cr = r3 % 8;
    const int n = ng * 8 + nr, c = cg * 8 + cr;
    const int t = (int)(blk / (K / kc)), g = (int)(blk % (K / kc));
    float val;
    if (!transpose)
        val = w[((long)t * cin + g * kc + c) * cout + n];
    else
        val = w[((long)(26 - t) * cin + n) * cout + g * kc + c];
    out[q] = __float2bfloat16_rn(val);
}

// Adam (Kingma and Ba, 2015) with bias correction, on FP32 master weights
__global__ void __launch_bounds__(kBlock) k_adam(long n, float* __restrict__ w, const float* __restrict__ g,
                                                 float* __restrict__ m, float* __restrict__ v, float lr, float b1,
                                                 float b2, float eps, float c1, float c2) {
    const long q = (long)blockIdx.x * blockDim.x + threadIdx.x;
    if (q >= n) return;
    const float gq = g[q];
    const float mq = b1 * m[q] + (1.f - b1) * gq;
    const float vq = b2 * v[q] + (1.f - b2) * gq * gq;
    m[q] = mq;
    v[q] = vq;
    w[q] -= lr * (mq / c1) / (sqrtf(vq / c2) + eps);
}

__global__ void __launch_bounds__(kBlock) k_to_float(long n, const double* __restrict__ x, double scale,
                                                     float* __restrict__ y) {
    const long q = (long)blockIdx.x * blockDim.x + threadIdx.x;
    if (q < n) y[q] = (float)(scale * x[q]);
}

__global__ void __launch_bounds__(kBlock) k_to_double(long n, const float* __restrict__ x, double scale,
                                                      double* __restrict__ y) {
    const long q = (long)blockIdx.x * blockDim.x + threadIdx.x;
    if (q < n) y[q] = scale * (double)x[q];
}

// partials of sum x^2 (FP64)
__global__ void __launch_bounds__(kBlock) k_sumsq(long n, const double* __restrict__ x, double* __restrict__ part) {
    __shared__ double sh[kBlock / 32];
    double a = 0.0;
    for (long q = (long)blockIdx.x * blockDim.x + threadIdx.x; q < n; q += (long)gridDim.x * blockDim.x)
        a += x[q] * x[q];
    for (int o = 16; o > 0; o >>= 1) a += __shfl_xor_sync(0xffffffffu, a, o);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (lane == 0) sh[warp] = a;
    __syncthreads();
    if (threadIdx.x == 0) {
        double s = 0.0;
        for (int q = 0; q < kBlock / 32; ++q) s += sh[q];
        part[blockIdx.x] = s;
    }
}

__global__ void k_sum_double(const double* __restrict__ part, int n, double* __restrict__ out) {
    if (threadIdx.x == 0 && blockIdx.x == 0) {
        double s = 0.0;
        for (int q = 0; q < n; ++q) s += part[q];
        *out = s;
    }
}

// r = sum over the (up to six) in-grid neighbours of (y_nb - y) + c * f:
// the h^2-scaled residual of the uniform-grid Neumann Laplacian for a
// network output y and the network input f (c: h^2 over the target scale)
__global__ void __launch_bounds__(kBlock) k_lap_residual(int n0, int n1, int n2, const float* __restrict__ y,
                                                         const float* __restrict__ f, float c, float* __restrict__ r) {
    const long V = (long)n0 * n1 * n2;
    const long v = (long)blockIdx.x * blockDim.x + threadIdx.x;
    if (v >= V) return;
    int i, j, k;
    decode(v, n1, n2, i, j, k);
    const float yc = y[v];
    float s = 0.f;
    if (i > 0) s += y[v - (long)n1 * n2] - yc;
    if (i < n0 - 1) s += y[v + (long)n1 * n2] - yc;
    if (j > 0) s += y[v - n2] - yc;
    if (j < n1 - 1) s += y[v + n2] - yc;
    if (k > 0) s += y[v - 1] - yc;
    if (k < n2 - 1) s += y[v + 1] - yc;
    r[v] = s + c * f[v];
}

// dy += w * (the same stencil applied to g): the adjoint of the residual's
// y-part, which is symmetric
__global__ void __launch_bounds__(kBlock) k_lap_add(int n0, int n1, int n2, const float* __restrict__ g, float w,
                                                    float* __restrict__ dy) {
    const long V = (long)n0 * n1 * n2;
    const long v = (long)blockIdx.x * blockDim.x + threadIdx.x;
    if (v >= V) return;
    int i, j, k;
    decode(v, n1, n2, i, j, k);
    const float gc = g[v];
    float s = 0.f;
    if (i > 0) s += g[v - (long)n1 * n2] - gc;
    if (i < n0 - 1) s += g[v + (long)n1 * n2] - gc;
    if (j > 0) s += g[v - n2] - gc;
    if (j < n1 - 1) s += g[v + n2] - gc;
    if (k > 0) s += g[v - 1] - gc;
    if (k < n2 - 1) s += g[v + 1] - gc;
    dy[v] += w * s;
}

inline unsigned blocks_for(long n) { return (unsigned)((n + kBlock - 1) / kBlock); }

}  // namespace

cudaError_t conv_in_launch(int n0, int n1, int n2, const float* x, const float* w, const float* b, bf16* out,
                           cudaStream_t s) {
    const long tiles = (long)((n2 + kInK - 1) / kInK) * ((n1 + kInJ - 1) / kInJ);
    // planes a CTA: those it walks, and about two more of start-up, times the
    // rounds of two CTAs an SM, at its least.  Eight on large grids; on small ones
    // a march of eight leaves SMs idle (16^3 31.0 -> 7.5 us, 64^3 33.7 -> 11.2,
    // 96^3 34.5 -> 31.0; a tile and plane a CTA without the ring took 10.5, 14.6, 43.3)
    int planes = kInI;
    long best = 0;
    for (int p = kInI; p >= 1; --p) {
        const long cost = (tiles * ((n0 + p - 1) / p) + 2 * kSms - 1) / (2 * kSms) * (p + 2);
        if (!best || cost < best) {
            best = cost;
            planes = p;
        }
    }
    const dim3 grid((unsigned)((n2 + kInK - 1) / kInK), (unsigned)((n1 + kInJ - 1) / kInJ),
                    (unsigned)((n0 + planes - 1) / planes));
    k_conv_in<<<grid, kBlock, 0, s>>>(n0, n1, n2, planes, x, w, b, out);
    return cudaGetLastError();
}

cudaError_t conv_in_wgrad_launch(int n0, int n1, int n2, const float* x, const bf16* dz, float* part, int nblocks,
                                 float* dw, cudaStream_t s) {
    const cudaError_t e =
        cudaFuncSetAttribute(k_conv_in_wgrad, cudaFuncAttributeMaxDynamicSharedMemorySize, kInTotals);
    if (e != cudaSuccess) return e;
    k_conv_in_wgrad<<<(unsigned)nblocks, kBlock, kInTotals, s>>>(n0, n1, n2, x, dz, part);
    k_sum_parts<<<blocks_for(28 * 16), kBlock, 0, s>>>(part, nblocks, 28 * 16, 28 * 16, 1.f, dw);
    return cudaGetLastError();
}

cudaError_t head_launch(long n, const bf16* d, const float* w, const float* b, float* y, cudaStream_t s) {
    k_head<<<blocks_for(n), kBlock, 0, s>>>(n, d, w, b, y);
    return cudaGetLastError();
}

cudaError_t head_grad_launch(long n, const bf16* d, const float* dy, const float* w, bf16* dz, float* part,
                             int nblocks, float* dw, cudaStream_t s) {
    k_head_grad<<<(unsigned)nblocks, kBlock, 0, s>>>(n, d, dy, w, dz, part);
    k_sum_parts<<<1, kBlock, 0, s>>>(part, nblocks, 17, 17, 1.f, dw);
    return cudaGetLastError();
}

cudaError_t pool_launch(int n0, int n1, int n2, int C, const bf16* src, bf16* dst, cudaStream_t s) {
    if (vec8({C}, {src, dst}) && (long)(n0 / 2) * (n1 / 2) * (n2 / 2) * (C / 8) < (1L << 32)) {
        k_pool8<<<blocks_for((long)(n0 / 2) * (n1 / 2) * (n2 / 2) * (C / 8)), kBlock, 0, s>>>(n0, n1, n2, C, src, dst);
        return cudaGetLastError();
    }
    k_pool<<<blocks_for((long)(n0 / 2) * (n1 / 2) * (n2 / 2) * (C / 2)), kBlock, 0, s>>>(n0, n1, n2, C, src, dst);
    return cudaGetLastError();
}

cudaError_t unpool_grad_launch(int n0, int n1, int n2, int ccat, int c0, const bf16* dcat, const bf16* act,
                               bf16* dz, cudaStream_t s) {
    if (vec8({ccat, c0}, {dcat, act, dz}) && (long)(n0 / 2) * (n1 / 2) * (n2 / 2) * (c0 / 8) < (1L << 32)) {
        k_unpool_grad8<<<blocks_for((long)(n0 / 2) * (n1 / 2) * (n2 / 2) * (c0 / 8)), kBlock, 0, s>>>(
            n0, n1, n2, ccat, c0, dcat, act, dz);
        return cudaGetLastError();
    }
    k_unpool_grad<<<blocks_for((long)(n0 / 2) * (n1 / 2) * (n2 / 2) * c0), kBlock, 0, s>>>(n0, n1, n2, ccat, c0,
                                                                                          dcat, act, dz);
    return cudaGetLastError();
}

cudaError_t skip_grad_launch(int n0, int n1, int n2, int ccat, int c0, int C, const bf16* dcat, const bf16* dp,
                             const bf16* src, bf16* dz, cudaStream_t s) {
    if (vec8({ccat, c0, C}, {dcat, dp, src, dz})) {
        k_skip_grad8<<<blocks_for((long)n0 * n1 * n2 * (C / 8)), kBlock, 0, s>>>(n0, n1, n2, ccat, c0, C, dcat, dp, src,
                                                                                 dz);
        return cudaGetLastError();
    }
    k_skip_grad<<<blocks_for((long)n0 * n1 * n2 * C), kBlock, 0, s>>>(n0, n1, n2, ccat, c0, C, dcat, dp, src, dz);
    return cudaGetLastError();
}

cudaError_t mse_launch(long n, const float* y, const float* t, float* dy, float* part, int nblocks, float* loss,
                       cudaStream_t s) {
    k_mse<<<(unsigned)nblocks, kBlock, 0, s>>>(n, y, t, dy, part);
    k_sum_parts<<<1, kBlock, 0, s>>>(part, nblocks, 1, 1, 1.f / (float)n, loss);
    return cudaGetLastError();
}

cudaError_t sum_parts_launch(const float* part, int nparts, long stride, long len, float* out, cudaStream_t s) {
    k_sum_parts<<<blocks_for(len), kBlock, 0, s>>>(part, nparts, stride, len, 1.f, out);
    return cudaGetLastError();
}

cudaError_t pack_launch(const float* w, int cin, int cout, int kc, int transpose, bf16* out, cudaStream_t s) {
    k_pack<<<blocks_for(27L * cin * cout), kBlock, 0, s>>>(w, cin, cout, kc, transpose, out);
    return cudaGetLastError();
}

cudaError_t adam_launch(long n, float* w, const float* g, float* m, float* v, float lr, float b1, float b2,
                        float eps, int step, cudaStream_t s) {
    const float c1 = 1.f - powf(b1, (float)step), c2 = 1.f - powf(b2, (float)step);
    k_adam<<<blocks_for(n), kBlock, 0, s>>>(n, w, g, m, v, lr, b1, b2, eps, c1, c2);
    return cudaGetLastError();
}

cudaError_t to_float_launch(long n, const double* x, double scale, float* y, cudaStream_t s) {
    k_to_float<<<blocks_for(n), kBlock, 0, s>>>(n, x, scale, y);
    return cudaGetLastError();
}

cudaError_t to_double_launch(long n, const float* x, double scale, double* y, cudaStream_t s) {
    k_to_double<<<blocks_for(n), kBlock, 0, s>>>(n, x, scale, y);
    return cudaGetLastError();
}

cudaError_t lap_residual_launch(int n0, int n1, int n2, const float* y, const float* f, float c, float* r,
                                cudaStream_t s) {
    k_lap_residual<<<blocks_for((long)n0 * n1 * n2), kBlock, 0, s>>>(n0, n1, n2, y, f, c, r);
    return cudaGetLastError();
}

cudaError_t lap_add_launch(int n0, int n1, int n2, const float* g, float w, float* dy, cudaStream_t s) {
    k_lap_add<<<blocks_for((long)n0 * n1 * n2), kBlock, 0, s>>>(n0, n1, n2, g, w, dy);
    return cudaGetLastError();
}

// ---- RMS normalisation with the scale kept on the device ---------------------
// (for a network queued inside a captured graph: no host round trip)
__global__ void __launch_bounds__(kBlock) k_sumsq32(long n, const float* __restrict__ x, double* __restrict__ part) {
    __shared__ double sh[kBlock / 32];
    double a = 0.0;
    for (long q = (long)blockIdx.x * blockDim.x + threadIdx.x; q < n; q += (long)gridDim.x * blockDim.x)
        a += (double)x[q] * (double)x[q];
    for (int o = 16; o > 0; o >>= 1) a += __shfl_xor_sync(0xffffffffu, a, o);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (lane == 0) sh[warp] = a;
    __syncthreads();
    if (threadIdx.x == 0) {
        double t = 0.0;
        for (int q = 0; q < kBlock / 32; ++q) t += sh[q];
        part[blockIdx.x] = t;
    }
}

// *rms = sqrt(sum of the parts / n), parts added in a fixed order
__global__ void k_rms_final(const double* __restrict__ part, int nparts, long n, double* rms) {
    double a = 0.0;
    for (int q = threadIdx.x; q < nparts; q += 32) a += part[q];
    for (int o = 16; o > 0; o >>= 1) a += __shfl_xor_sync(0xffffffffu, a, o);
    if (threadIdx.x == 0) *rms = sqrt(a / (double)n);
}

// y = sign * x / rms (zero when rms is zero)
__global__ void k_div_rms(long n, const float* __restrict__ x, float sign, const double* __restrict__ rms,
                          float* __restrict__ y) {
    const double r = *rms;
    const float f = r > 0.0 ? (float)(sign / r) : 0.f;
    for (long q = (long)blockIdx.x * blockDim.x + threadIdx.x; q < n; q += (long)gridDim.x * blockDim.x)
        y[q] = f * x[q];
}

// x = y * scale * rms
__global__ void k_mul_rms(long n, const float* __restrict__ y, double scale, const double* __restrict__ rms,
                          float* __restrict__ x) {
    const float f = (float)(scale * *rms);
    for (long q = (long)blockIdx.x * blockDim.x + threadIdx.x; q < n; q += (long)gridDim.x * blockDim.x)
        x[q] = f * y[q];
}

cudaError_t rms_normalise_launch(long n, const float* x, float sign, double* part, int nblocks, double* rms,
                                 float* y, cudaStream_t s) {
    k_sumsq32<<<(unsigned)nblocks, kBlock, 0, s>>>(n, x, part);
    k_rms_final<<<1, 32, 0, s>>>(part, nblocks, n, rms);
    k_div_rms<<<blocks_for(n), kBlock, 0, s>>>(n, x, sign, rms, y);
    return cudaGetLastError();
}

cudaError_t rms_restore_launch(long n, const float* y, double scale, const double* rms, float* x, cudaStream_t s) {
    k_mul_rms<<<blocks_for(n), kBlock, 0, s>>>(n, y, scale, rms, x);
    return cudaGetLastError();
}

cudaError_t sumsq_launch(long n, const double* x, double* part, int nblocks, double* out, cudaStream_t s) {
    k_sumsq<<<(unsigned)nblocks, kBlock, 0, s>>>(n, x, part);
    k_sum_double<<<1, 32, 0, s>>>(part, nblocks, out);
    return cudaGetLastError();
}

}  // namespace bun
