// bun_conv.cu -- 3x3x3 convolutions of the U-Net as implicit GEMMs on the
// sm_100a tensor cores (tcgen05.mma kind::f16, BF16 operands, FP32
// accumulators in tensor memory).
//
// Forward and data-gradient kernel (k_conv): one CTA computes a tile of 128
// consecutive voxels x all output channels.  GEMM view: M = voxels, N =
// output channels, K = 27 taps x input channels, walked in stages of one tap
// and KC channels.  Warps 0-3 load the stages with cp.async (the A tile is
// the tile's voxels shifted by the tap, zero-filled outside the grid; the B
// tile is a contiguous block of the packed weights) and signal a full
// barrier per stage; one thread of warp 4 issues KC/16 MMAs per stage and
// releases the stage through tcgen05.commit; after the last stage warps 0-3
// read the accumulator rows from tensor memory (thread = voxel = TMEM lane)
// and apply bias, ReLU or a ReLU mask before storing BF16.
//
// Weight-gradient kernel (k_wgrad): GEMM view M = (tap, input channel) rows
// in tiles of 128, N = output channels, K = voxels; both operands are read
// MN-major (channels contiguous), which is the channels-last layout of the
// activations, so the A tile is 16 row groups of 8 channels x 128 voxels of
// the tap-shifted input and the B tile the matching 128 voxels of the output
// gradient.  K is split over grid.y; each split writes FP32 partial sums
// that a CUDA-core kernel adds in a fixed order.
//
// Convolutions of 16 to 64 output channels march along j instead (k_conv_rows,
// below), and weight gradients on rows of whole 16-voxel groups take blocks of
// rows (k_wgrad_rows): a row is loaded once for the taps that need it.
//
// Shared-memory operand layouts are the canonical no-swizzle (interleaved)
// ones of the tcgen05 matrix descriptors: a core matrix is 8 rows of 16
// bytes (128 contiguous bytes).  K-major tiles: a row is one M/N index with
// 8 consecutive K elements; core matrices 128 bytes apart along K (leading
// byte offset) and one row group apart along M/N (stride byte offset).
// MN-major tiles: a row is one K index with 8 consecutive M/N elements; core
// matrices 128 bytes apart along K (leading) and 2 KB apart along M/N
// (stride).
//
// Every wait on a barrier is bounded (about two seconds of SM clock); a
// thread that gives up records kErrTimeout, stops issuing work, and the CTA
// still waits for its issued MMAs before freeing tensor memory.

#include "bun_internal.h"

#include <algorithm>

namespace bun {

namespace {

constexpr int kTile = 128;       // voxels per conv tile / per wgrad K block
constexpr int kProducers = 128;  // warps 0-3: loads, then the epilogue
constexpr int kThreads = 160;    // + warp 4: TMEM allocation and MMA issue
constexpr long long kWaitCycles = 4000000000LL;

__device__ __forceinline__ uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

__device__ __forceinline__ void mbar_init(uint64_t* bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count) : "memory");
}

__device__ __forceinline__ bool mbar_test(uint64_t* bar, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(smem_u32(bar)), "r"(parity)
        : "memory");
    return ok != 0;
}

// wait until the phase with this parity has completed; false on timeout
__device__ __forceinline__ bool mbar_wait(uint64_t* bar, uint32_t parity) {
    if (mbar_test(bar, parity)) return true;
    const long long t0 = clock64();
    while (!mbar_test(bar, parity))
        if (clock64() - t0 > kWaitCycles) return false;
    return true;
}

// 16-byte global -> shared copy; zero-filled when !valid (src is not read)
__device__ __forceinline__ void cp16(uint32_t dst, const void* src, bool valid) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(valid ? 16 : 0)
                 : "memory");
}

// arrive on the barrier once this thread's cp.async copies have landed
__device__ __forceinline__ void cp_arrive(uint64_t* bar) {
    asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];" ::"r"(smem_u32(bar)) : "memory");
}

__device__ __forceinline__ void tc_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }

// whole warp
__device__ __forceinline__ void tmem_alloc(uint32_t* slot, uint32_t ncols) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(slot)),
                 "r"(ncols)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}

__device__ __forceinline__ void tmem_free(uint32_t taddr, uint32_t ncols) {
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(ncols) : "memory");
}

// no-swizzle shared-memory matrix descriptor (version 1)
__device__ __forceinline__ uint64_t sdesc(uint32_t addr, uint32_t lbo, uint32_t sbo) {
    return (uint64_t)((addr >> 4) & 0x3FFFu) | ((uint64_t)((lbo >> 4) & 0x3FFFu) << 16) |
           ((uint64_t)((sbo >> 4) & 0x3FFFu) << 32) | (1ull << 46);
}

// instruction descriptor: BF16 x BF16 -> FP32, M x N, operand majorness
__host__ __device__ constexpr uint32_t idesc_bf16(int m, int n, bool a_mn, bool b_mn) {
    return (1u << 4) | (1u << 7) | (1u << 10) | ((a_mn ? 1u : 0u) << 15) | ((b_mn ? 1u : 0u) << 16) |
           ((uint32_t)(n >> 3) << 17) | ((uint32_t)(m >> 4) << 24);
}

__device__ __forceinline__ void umma(uint32_t d, uint64_t adesc, uint64_t bdesc, uint32_t idesc, uint32_t acc) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(d),
        "l"(adesc), "l"(bdesc), "r"(idesc), "r"(acc)
        : "memory");
}

// arrive on the barrier when every MMA issued so far has completed
__device__ __forceinline__ void umma_commit(uint64_t* bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(
                     smem_u32(bar))
                 : "memory");
}

// 16 consecutive FP32 columns of this thread's TMEM lane
__device__ __forceinline__ void tmem_ld16(uint32_t taddr, float* v) {
    uint32_t r[16];
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, "
        "%14, %15}, [%16];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
          "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
        : "r"(taddr));
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
    for (int q = 0; q < 16; ++q) v[q] = __uint_as_float(r[q]);
}

// the 8-channel chunk starting at channel ch of full-resolution voxel
// (i, j, k) of the (possibly concatenated, possibly upsampled) input
__device__ __forceinline__ const bf16* in_ptr(const ConvIn& in, int n1, int n2, int i, int j, int k, int ch) {
    if (ch < in.c0) {
        if (in.up0) {
            i >>= 1;
            j >>= 1;
            k >>= 1;
            n1 >>= 1;
            n2 >>= 1;
        }
        return in.src0 + (((long)i * n1 + j) * n2 + k) * in.c0 + ch;
    }
    return in.src1 + (((long)i * n1 + j) * n2 + k) * in.c1 + (ch - in.c0);
}

template <int NOUT>
__host__ __device__ constexpr int tmem_cols() {
    return NOUT <= 32 ? 32 : NOUT <= 64 ? 64 : NOUT <= 128 ? 128 : 256;
}

// ---------------------------------------------------------------------------
// forward / data-gradient convolution
// ---------------------------------------------------------------------------
template <int KC, int NOUT, int S>
__global__ void __launch_bounds__(kThreads) k_conv(ConvArgs a) {
    constexpr int A_BYTES = kTile * KC * 2;
    constexpr int B_BYTES = NOUT * KC * 2;
    constexpr int STAGE = A_BYTES + B_BYTES;
    constexpr uint32_t NCOLS = tmem_cols<NOUT>();
    extern __shared__ __align__(1024) uint8_t smem[];
    uint64_t* full = reinterpret_cast<uint64_t*>(smem + S * STAGE);
    uint64_t* empty = full + S;
    uint64_t* accb = empty + S;
    uint32_t* slot = reinterpret_cast<uint32_t*>(accb + 1);

    const int tid = threadIdx.x, warp = tid >> 5;
    const int n0 = a.n0, n1 = a.n1, n2 = a.n2;
    const int nq = (a.in.c0 + a.in.c1) / KC;
    const int iters = 27 * nq;
    const long V = (long)n0 * n1 * n2;
    const long v = (long)blockIdx.x * kTile + (tid & (kTile - 1));

    if (tid == 0) {
        for (int s = 0; s < S; ++s) {
            mbar_init(&full[s], kProducers);
            mbar_init(&empty[s], 1);
        }
        mbar_init(accb, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 4) tmem_alloc(slot, NCOLS);
    tc_before();
    __syncthreads();
    tc_after();
    const uint32_t tmem = *slot;
    bool ok = true;

    if (warp < 4) {
        // ---- producers: one voxel row of every A tile, a share of the B tile
        const bool row = v < V;
        int i = 0, j = 0, k = 0;
        if (row) {
            k = (int)(v % n2);
            const long q = v / n2;
            j = (int)(q % n1);
            i = (int)(q / n1);
        }
        const uint32_t a_off = (uint32_t)(tid >> 3) * (KC * 16) + (uint32_t)(tid & 7) * 16;
        const uint32_t base = smem_u32(smem);
        for (int it = 0; it < iters; ++it) {
            const int s = it % S;
            const uint32_t use = (uint32_t)(it / S);
            if (!mbar_wait(&empty[s], (use & 1) ^ 1)) {
                ok = false;
                break;
            }
            const int t = it / nq, qq = it - t * nq;
            const int ii = i + t / 9 - 1, jj = j + (t / 3) % 3 - 1, kk = k + t % 3 - 1;
            const bool valid = row && ii >= 0 && ii < n0 && jj >= 0 && jj < n1 && kk >= 0 && kk < n2;
            const bf16* src = valid ? in_ptr(a.in, n1, n2, ii, jj, kk, qq * KC) : a.wpack;
            const uint32_t As = base + s * STAGE;
#pragma unroll
            for (int h = 0; h < KC / 8; ++h) cp16(As + a_off + h * 128, src + (valid ? h * 8 : 0), valid);
            const bf16* w = a.wpack + (long)it * (NOUT * KC);
            const uint32_t Bs = As + A_BYTES;
            for (int c = tid; c < NOUT * KC / 8; c += kProducers) cp16(Bs + c * 16, w + c * 8, true);
            cp_arrive(&full[s]);
        }
    } else if (tid == kProducers) {
        // ---- MMA issue: KC/16 MMAs of 128 x NOUT x 16 per stage
        constexpr uint32_t idesc = idesc_bf16(kTile, NOUT, false, false);
        const uint32_t base = smem_u32(smem);
        for (int it = 0; it < iters; ++it) {
            const int s = it % S;
            const uint32_t use = (uint32_t)(it / S);
            if (!mbar_wait(&full[s], use & 1)) {
                ok = false;
                break;
            }
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            tc_after();
            const uint32_t As = base + s * STAGE, Bs = As + A_BYTES;
#pragma unroll
            for (int q = 0; q < KC / 16; ++q)
                umma(tmem, sdesc(As + q * 256, 128, KC * 16), sdesc(Bs + q * 256, 128, KC * 16), idesc,
                     (it | q) != 0);
            umma_commit(&empty[s]);
        }
        umma_commit(accb);
    }

    if (warp < 4) {
        // ---- epilogue: thread = voxel = TMEM lane
        bool done = mbar_wait(accb, 0);
        done = __all_sync(0xffffffffu, done);
        tc_after();
        if (!done) ok = false;
        if (done) {
            const bool row = v < V;
#pragma unroll 1
            for (int c0 = 0; c0 < NOUT; c0 += 16) {
                float acc[16];
                tmem_ld16(tmem + ((uint32_t)(warp * 32) << 16) + (uint32_t)c0, acc);
                if (!row) continue;
                if (a.bias) {
#pragma unroll
                    for (int q = 0; q < 16; ++q) acc[q] += a.bias[c0 + q];
                }
                if (a.relu) {
#pragma unroll
                    for (int q = 0; q < 16; ++q) acc[q] = fmaxf(acc[q], 0.f);
                }
                if (a.mask) {
                    const uint4* mp = reinterpret_cast<const uint4*>(a.mask + v * NOUT + c0);
                    uint4 mv[2] = {mp[0], mp[1]};
                    const bf16* m = reinterpret_cast<const bf16*>(mv);
#pragma unroll
                    for (int q = 0; q < 16; ++q)
                        if (!(__bfloat162float(m[q]) > 0.f)) acc[q] = 0.f;
                }
                uint4 ov[2];
                __nv_bfloat162* o = reinterpret_cast<__nv_bfloat162*>(ov);
#pragma unroll
                for (int q = 0; q < 8; ++q) o[q] = __floats2bfloat162_rn(acc[2 * q], acc[2 * q + 1]);
                uint4* op = reinterpret_cast<uint4*>(a.out + v * NOUT + c0);
                op[0] = ov[0];
                op[1] = ov[1];
            }
        }
    }

    if (!ok && a.err) atomicExch(a.err, kErrTimeout);
    tc_before();
    __syncthreads();
    if (warp == 4) {
        tc_after();
        mbar_wait(accb, 0);  // no MMA may still write the accumulator
        tmem_free(tmem, NCOLS);
    }
}

// ---------------------------------------------------------------------------
// weight gradient
// ---------------------------------------------------------------------------
template <int NOUT, int S>
__global__ void __launch_bounds__(kThreads) k_wgrad(WgradArgs a) {
    constexpr int A_BYTES = 128 * kTile * 2;  // 16 row groups x 16 voxel groups x 128 B
    constexpr int B_BYTES = NOUT * kTile * 2;
    constexpr int STAGE = A_BYTES + B_BYTES;
    constexpr uint32_t NCOLS = tmem_cols<NOUT>();
    extern __shared__ __align__(1024) uint8_t smem[];
    uint64_t* full = reinterpret_cast<uint64_t*>(smem + S * STAGE);
    uint64_t* empty = full + S;
    uint64_t* accb = empty + S;
    uint32_t* slot = reinterpret_cast<uint32_t*>(accb + 1);

    const int tid = threadIdx.x, warp = tid >> 5;
    const int n0 = a.n0, n1 = a.n1, n2 = a.n2;
    const int cin = a.in.c0 + a.in.c1;
    const long V = (long)n0 * n1 * n2;
    const long nblk = (V + kTile - 1) / kTile;
    const int split = blockIdx.y;
    const int iters = split < nblk ? (int)((nblk - 1 - split) / a.nsplit + 1) : 0;
    const int mt = blockIdx.x;

    if (tid == 0) {
        for (int s = 0; s < S; ++s) {
            mbar_init(&full[s], kProducers);
            mbar_init(&empty[s], 1);
        }
        mbar_init(accb, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 4) tmem_alloc(slot, NCOLS);
    tc_before();
    __syncthreads();
    tc_after();
    const uint32_t tmem = *slot;
    bool ok = true;

    if (warp < 4) {
        // the 16 row groups of this M tile: tap offset and first channel
        int gdi[16], gdj[16], gdk[16], gch[16];
        bool gon[16];
#pragma unroll
        for (int g = 0; g < 16; ++g) {
            const int r0 = mt * 128 + g * 8;
            const int t = r0 / cin;
            gon[g] = r0 < a.rows;
            gch[g] = r0 - t * cin;
            gdi[g] = t / 9 - 1;
            gdj[g] = (t / 3) % 3 - 1;
            gdk[g] = t % 3 - 1;
        }
        const uint32_t off = (uint32_t)(tid >> 3) * 128 + (uint32_t)(tid & 7) * 16;
        const uint32_t base = smem_u32(smem);
        for (int it = 0; it < iters; ++it) {
            const int s = it % S;
            const uint32_t use = (uint32_t)(it / S);
            if (!mbar_wait(&empty[s], (use & 1) ^ 1)) {
                ok = false;
                break;
            }
            const long v = ((long)split + (long)it * a.nsplit) * kTile + tid;
            const bool row = v < V;
            int i = 0, j = 0, k = 0;
            if (row) {
                k = (int)(v % n2);
                const long q = v / n2;
                j = (int)(q % n1);
                i = (int)(q / n1);
            }
            const uint32_t As = base + s * STAGE, Bs = As + A_BYTES;
#pragma unroll
            for (int g = 0; g < 16; ++g) {
                const int ii = i + gdi[g], jj = j + gdj[g], kk = k + gdk[g];
                const bool valid = row && gon[g] && ii >= 0 && ii < n0 && jj >= 0 && jj < n1 && kk >= 0 && kk < n2;
                const bf16* src = valid ? in_ptr(a.in, n1, n2, ii, jj, kk, gch[g]) : a.dz;
                cp16(As + g * 2048 + off, src, valid);
            }
#pragma unroll
            for (int g = 0; g < NOUT / 8; ++g) cp16(Bs + g * 2048 + off, row ? a.dz + v * NOUT + g * 8 : a.dz, row);
            cp_arrive(&full[s]);
        }
    } else if (tid == kProducers) {
        constexpr uint32_t idesc = idesc_bf16(128, NOUT, true, true);
        const uint32_t base = smem_u32(smem);
        for (int it = 0; it < iters; ++it) {
            const int s = it % S;
            const uint32_t use = (uint32_t)(it / S);
            if (!mbar_wait(&full[s], use & 1)) {
                ok = false;
                break;
            }
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            tc_after();
            const uint32_t As = base + s * STAGE, Bs = As + A_BYTES;
#pragma unroll
            for (int q = 0; q < kTile / 16; ++q)
                umma(tmem, sdesc(As + q * 256, 128, 2048), sdesc(Bs + q * 256, 128, 2048), idesc, (it | q) != 0);
            umma_commit(&empty[s]);
        }
        umma_commit(accb);
    }

    if (warp < 4) {
        bool done = mbar_wait(accb, 0);
        done = __all_sync(0xffffffffu, done);
        tc_after();
        if (!done) ok = false;
        if (done) {
            float* dst = a.part + ((long)split * a.rows_pad + (long)mt * 128 + tid) * NOUT;
#pragma unroll 1
            for (int c0 = 0; c0 < NOUT; c0 += 16) {
                float acc[16];
                tmem_ld16(tmem + ((uint32_t)(warp * 32) << 16) + (uint32_t)c0, acc);
                if (iters == 0) {
#pragma unroll
                    for (int q = 0; q < 16; ++q) acc[q] = 0.f;  // nothing was accumulated
                }
#pragma unroll
                for (int q = 0; q < 16; q += 4)
                    *reinterpret_cast<float4*>(dst + c0 + q) = make_float4(acc[q], acc[q + 1], acc[q + 2], acc[q + 3]);
            }
        }
    }

    if (!ok && a.err) atomicExch(a.err, kErrTimeout);
    tc_before();
    __syncthreads();
    if (warp == 4) {
        tc_after();
        mbar_wait(accb, 0);
        tmem_free(tmem, NCOLS);
    }
}

// ---------------------------------------------------------------------------
// weight gradient by blocks of rows (n2 % 16 == 0, channels in blocks of 16)
// ---------------------------------------------------------------------------
// k_wgrad gathers the 128 voxels of a K block once for every (tap, channel)
// row tile, 27 times over, and its loads bound it (48 -> 16 channels at 128^3:
// 1.94 ms, tensor pipe idle).  Here a CTA owns one plane offset di and 16 input
// channels and takes blocks of W = 128 / COUT rows j of the output gradient
// (plane i, 128 voxels along k) with the W + 2 input rows of plane i + di that
// meet them:
//   M = (output-gradient row, output channel), N = (input row, input channel),
//   K = voxels,
// one MMA chain per tap offset dk -- a shift of the input rows' start address,
// as in k_conv_rows.  M is full (an MMA costs its 128 rows' operand, whatever
// they hold); of the products those of rows j and j-1 .. j+1 are wanted, the
// diagonal blocks, which is 3 W of W (W + 2).  One input row against the three
// rows that meet it filled 48 of the 128 rows of M for 16 channels and was bound
// by the tensor pipe: five times as many MMA cycles a row.
// Rows outside the grid are zero.  Both operands are MN-major: chunks of 8
// channels x voxels of 16 bytes.
// D: lane = (row, output channel), column = (dk, input row, input channel),
// added up over all blocks of the split.  At the end the W diagonals are added
// in order by way of shared memory and written once, as k_wgrad's partials.
// Measured, us, k_wgrad / one input row at a time / now: at 128^3 48 -> 16
// channels 1936 / 663 / 292, 16 -> 16 735 / 250 / 119; at 64^3 96 -> 32
// 802 / 210 / 162, 32 -> 32 286 / 78 / 61, 16 -> 32 160 / 72 / 40; k_wgrad / now:
// at 32^3 128 -> 64 150 / 74, 64 -> 64 90 / 42; at 16^3 64 -> 64 27 / 17.  Bound
// by the blocks' supply (74 KB against 24 MMAs): 48 -> 16 at 128^3 has the tensor
// pipe active 39 %, L1 51 %, and its warps wait for the loads; 64 -> 64 there, two
// stages, has L1 at 95 %.
constexpr int kWgVox = 128;                      // voxels of a block's rows
constexpr int kWgInChunk = (kWgVox + 2) * 16;    // bytes of 8 input channels of a row (k0-1 .. k0+128)
constexpr int kWgDzChunk = kWgVox * 16;          // bytes of 8 output channels of a row

template <int COUT>
struct WgRowShape {
    static constexpr int W = 128 / COUT;                    // rows of a block
    static constexpr int N = (W + 2) * 16;
    static constexpr int DZ = W * (COUT / 8) * kWgDzChunk;
    static constexpr int STAGE = DZ + (W + 2) * 2 * kWgInChunk;
    // three stages and one CTA an SM; 64 channels: two and two
    static constexpr int S = COUT == 64 ? 2 : 3;
    static constexpr uint32_t NCOLS = 3 * N <= 256 ? 256 : 512;
    static constexpr int smem = S * STAGE + (2 * S + 1) * 8 + 16;
    static_assert(W * 9 * 16 * COUT * 4 <= S * STAGE, "the diagonals take the stages' place");
};

template <int COUT>
__global__ void __launch_bounds__(kThreads) k_wgrad_rows(WgradArgs a) {
    using F = WgRowShape<COUT>;
    constexpr int S = F::S, W = F::W, N = F::N;
    extern __shared__ __align__(1024) uint8_t smem[];
    uint64_t* full = reinterpret_cast<uint64_t*>(smem + S * F::STAGE);
    uint64_t* empty = full + S;
    uint64_t* accb = empty + S;
    uint32_t* slot = reinterpret_cast<uint32_t*>(accb + 1);

    const int tid = threadIdx.x, warp = tid >> 5;
    const int n0 = a.n0, n1 = a.n1, n2 = a.n2;
    const int split = blockIdx.x, di = blockIdx.y, cb = blockIdx.z * 16;
    const int nks = (n2 + kWgVox - 1) / kWgVox, njs = (n1 + W - 1) / W;
    const int units = n0 * nks * njs;

    if (tid == 0) {
        for (int r = 0; r < S; ++r) {
            mbar_init(&full[r], kProducers);
            mbar_init(&empty[r], 1);
        }
        mbar_init(accb, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 4) tmem_alloc(slot, F::NCOLS);
    tc_before();
    __syncthreads();
    tc_after();
    const uint32_t tmem = *slot;
    const uint32_t base = smem_u32(smem);
    bool ok = true, any = false;

    // a block's plane, first voxel and row, and voxels; false where the input
    // plane lies outside the grid
    auto unit = [&](int un, int& i, int& k0, int& js, int& kv) {
        const int ks = un % nks, q = un / nks;
        k0 = ks * kWgVox;
        kv = min(kWgVox, n2 - k0);
        js = (q % njs) * W;
        i = q / njs;
        const int ii = i + di - 1;
        return ii >= 0 && ii < n0;
    };

    if (warp < 4) {
        // ---- loader; the sources of the two chunks of channels
        const bf16* src[2];
        int cs[2], up[2];
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const int ch = cb + h * 8;
            const bool first = ch < a.in.c0;
            src[h] = first ? a.in.src0 + ch : a.in.src1 + (ch - a.in.c0);
            cs[h] = first ? a.in.c0 : a.in.c1;
            up[h] = first ? a.in.up0 : 0;
        }
        int e = 0;
        for (int un = split; ok && un < units; un += a.nsplit) {
            int i, k0, js, kv;
            if (!unit(un, i, k0, js, kv)) continue;
            const int ii = i + di - 1, r = e % S;
            if (!mbar_wait(&empty[r], ((uint32_t)(e / S) & 1) ^ 1)) {
                ok = false;
                break;
            }
            ++e;
            const uint32_t st = base + r * F::STAGE;
            // 2^lg voxels by 128 / 2^lg rows at once
            const int lg = kv > 64 ? 7 : kv > 32 ? 6 : kv > 16 ? 5 : 4;
            const int v = tid & ((1 << lg) - 1), w0 = tid >> lg, ws = kProducers >> lg;
            if (v < kv) {
                const bf16* dp = a.dz + (((long)i * n1 + js) * n2 + k0 + v) * COUT;
                const uint32_t d0 = st + v * 16, i0 = st + F::DZ + (v + 1) * 16;
                const bf16* p[2];
                for (int h = 0; h < 2; ++h)
                    p[h] = src[h] + ((long)(ii >> up[h]) * (n1 >> up[h]) * (n2 >> up[h]) + ((k0 + v) >> up[h])) * cs[h];
#pragma unroll 2
                for (int w = w0; w < W; w += ws) {
                    const bool valid = js + w < n1;
#pragma unroll
                    for (int h = 0; h < COUT / 8; ++h)
                        cp16(d0 + (w * (COUT / 8) + h) * kWgDzChunk, valid ? dp + (long)w * n2 * COUT + h * 8 : a.dz, valid);
                }
#pragma unroll 2
                for (int w = w0; w < W + 2; w += ws) {
                    const int jj = js - 1 + w;
                    const bool valid = jj >= 0 && jj < n1;
#pragma unroll
                    for (int h = 0; h < 2; ++h)
                        cp16(i0 + (w * 2 + h) * kWgInChunk,
                             valid ? p[h] + (long)((jj >> up[h]) * (n2 >> up[h])) * cs[h] : a.dz, valid);
                }
            }
            // the voxels before and behind the rows
            if (tid < 2 * (W + 2)) {
                const int w = tid >> 1, jj = js - 1 + w, k = tid & 1 ? k0 + kv : k0 - 1;
                const bool valid = jj >= 0 && jj < n1 && k >= 0 && k < n2;
                const uint32_t d = st + F::DZ + w * 2 * kWgInChunk + (tid & 1 ? kv + 1 : 0) * 16;
#pragma unroll
                for (int h = 0; h < 2; ++h)
                    cp16(d + h * kWgInChunk, valid ? in_ptr(a.in, n1, n2, ii, jj, k, cb + h * 8) : a.dz, valid);
            }
            cp_arrive(&full[r]);
        }
    } else if (tid == kProducers) {
        // ---- MMA issue: per block and dk, kv / 16 MMAs of 128 x N x 16
        constexpr uint32_t idesc = idesc_bf16(128, N, true, true);
        int e = 0;
        for (int un = split; ok && un < units; un += a.nsplit) {
            int i, k0, js, kv;
            if (!unit(un, i, k0, js, kv)) continue;
            if (!mbar_wait(&full[e % S], (uint32_t)(e / S) & 1)) {
                ok = false;
                break;
            }
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            tc_after();
            const uint32_t as = base + (uint32_t)(e % S) * F::STAGE, bs = as + F::DZ;
#pragma unroll 1
            for (int dk = 0; dk < 3; ++dk)
#pragma unroll 1
                for (int q = 0; q < kv / 16; ++q)
                    umma(tmem + dk * N, sdesc(as + q * 256, 128, kWgDzChunk),
                         sdesc(bs + dk * 16 + q * 256, 128, kWgInChunk), idesc, any || q != 0);
            any = true;
            umma_commit(&empty[e % S]);
            ++e;
        }
        umma_commit(accb);
    }

    if (warp < 4) {
        for (int un = split; !any && un < units; un += a.nsplit) {
            int i, k0, js, kv;
            any = unit(un, i, k0, js, kv);
        }
        bool done = mbar_wait(accb, 0);
        done = __all_sync(0xffffffffu, done);
        tc_after();
        if (!done) ok = false;
        // lane = (row r, output channel n) met input row r + dj: every stage has
        // been read, the diagonals go where they were
        float* red = reinterpret_cast<float*>(smem);
        const int r = tid / COUT, n = tid % COUT, r0 = warp * 32 / COUT;
        constexpr int T = COUT < 32 ? 4 : 3;  // input rows that meet a row of the warp
        if (done && any) {
#pragma unroll 1
            for (int dk = 0; dk < 3; ++dk)
#pragma unroll 1
                for (int t = 0; t < T; ++t) {
                    float acc[16];
                    tmem_ld16(tmem + ((uint32_t)(warp * 32) << 16) + (uint32_t)(dk * N + (r0 + t) * 16), acc);
                    const int dj = r0 + t - r;
                    if (dj >= 0 && dj < 3) {
                        float* dst = red + ((r * 9 + dj * 3 + dk) * 16) * COUT + n;
#pragma unroll
                        for (int q = 0; q < 16; ++q) dst[q * COUT] = acc[q];
                    }
                    __syncwarp();
                }
        }
        asm volatile("bar.sync 1, 128;" ::: "memory");
        const int C = a.in.c0 + a.in.c1;
        if (done) {
            for (int x = tid; x < 9 * 16 * COUT; x += kProducers) {
                float sum = 0.f;
                if (any) {
#pragma unroll
                    for (int w = 0; w < W; ++w) sum += red[w * 9 * 16 * COUT + x];
                }
                const int c = x / COUT % 16, tap = x / (16 * COUT);
                a.part[((long)split * a.rows_pad + (di * 9 + tap) * C + cb + c) * COUT + x % COUT] = sum;
            }
        }
    }

    if (!ok && a.err) atomicExch(a.err, kErrTimeout);
    tc_before();
    __syncthreads();
    if (warp == 4) {
        tc_after();
        mbar_wait(accb, 0);  // no MMA may still write the accumulator
        tmem_free(tmem, F::NCOLS);
    }
}

// ---------------------------------------------------------------------------
// forward / data-gradient convolution marching along j
// ---------------------------------------------------------------------------
// A CTA owns 128 positions of a plane (fixed j) of the grid and JS rows j, and
// walks the input rows jj = js-1 .. je, each loaded once by cp.async into a
// ring.  A position of row jj and its neighbours (di, dk) lie P di + dk apart in
// the loaded run, one of two ways:
//   n2 % 128 == 0  128 voxels k0 .. k0+127 of plane i, the run being the three
//                  rows i-1 .. i+1 over k0-1 .. k0+128 (P = 130);
//   else           a stretch of the planes' rows one behind another with one
//                  zero voxel between them, the halo of both (P = n2 + 1), so
//                  short rows fill the 128 positions too.
// The run is laid out as [8-channel chunk h][position] x 16 bytes.  The A operand
// of (di, dk) and channels 16u .. 16u+15 is then a K-major no-swizzle matrix
// starting at chunk 2u, position P di + dk, with the chunks' distance as
// leading and 128 bytes (8 positions) as stride byte offset: a tap is a change
// of start address.
// With 16 to 48 output channels an MMA costs what its A operand's 4 KB cost,
// whatever N is, so the three dj of (di, dk) are one
// MMA: the input row's products for output rows jj-1, jj and jj+1, whose
// accumulators are neighbours in tensor memory (JS rows' are there, zeroed
// at the start), with the weights of dj = 2, 1, 0 side by side as B.
// Input channels go in groups of CG: the CTA walks its rows, JS at most, once per
// group with that group's weights (two buffers, the next group's load under this
// one's MMAs); the sums stay in FP32 in tensor memory from the first group to
// the last.  With one group a row is complete after its three input rows, and the
// CTA may walk more (RING): the epilogue zeroes a row's accumulator for the JS-th
// row after it, and where the three rows' accumulators begin again they take two
// MMAs.
// Warps 0-3: epilogue (thread = position = TMEM lane), a row as soon as the
// last group completes it; warps 4-7: loader; warp 8: TMEM allocation, one
// thread issues the MMAs.
// Measured against a tap an MMA on the n2 % 128 == 0 rows, the only ones that
// marched, and against k_conv elsewhere (256^3 network, cin -> nout at the
// level's size, us before / now; the tensor pipe is active 18 to 40 % of the time,
// L1 47 to 57 %: the rows' supply and the hand-over between the warps bound it):
//   256^3  16 -> 16   663 /  547     48 -> 16   3359 / 1282
//   128^3  96 -> 32  2869 /  418     32 -> 32   360 /  191     16 -> 32  132 / 103
//    64^3  32 -> 64   119 /   47     64 -> 64    319 /   76   128 -> 64  589 / 134
//    32^3  64 -> 64    50 /   21;  16^3 64 -> 64   30 /   17
constexpr int kRowThreads = 288;
constexpr int kRowRing = 8;  // most rows of the ring
constexpr int kRowsMost = 32;  // most rows j a CTA

struct RowPlan {
    int P;       // distance of the planes' rows in the run
    int nvox;    // positions of the run: 2 P + 130
    int nr;      // rows of the ring
    int nw;      // weight buffers: two, one where there is one group of channels
    int rows;    // rows j a CTA; at most JS but with RING
    int lk;      // log2 of the 8-channel chunks of a packed weight block
    int ntot;    // output channels, NOUT of them a CTA (blockIdx.y)
    int stream;  // rows one behind another
    int tiles;   // of 128 positions; CTA = segment * tiles + tile
};

template <int CG, int NOUT, int JS>
struct RowShape {
    static constexpr int WBYTES = 27 * CG * NOUT * 2;
    static constexpr uint32_t NCOLS = JS * NOUT <= 256 ? 256 : 512;
    static constexpr int BARS = (2 * kRowRing + 4 + 2 * JS + 1) * 8 + 16;
    // longest run: P of 256 (or 130; groups of 32 have rows below 128 only)
    static constexpr int MAXVOX = CG == 16 ? 2 * 256 + kTile + 2 : 2 * 130 + kTile + 2;
    static_assert(JS * NOUT <= 512 && 3 * NOUT <= 256, "tensor memory");
};

// the plane and voxel of a position of tile's run (q = 0: one row and one voxel
// before its first position); false outside the grid
__device__ __forceinline__ bool row_voxel(const ConvArgs& a, const RowPlan& R, int tile, int q, int& i, int& k) {
    if (R.stream) {
        // counted from the voxel before the plane before the first
        const unsigned g = (unsigned)tile * kTile + (unsigned)q, r = g ? (g - 1) / (unsigned)R.P : 0;
        i = g ? (int)r - 1 : -1;
        k = (int)(g - 1 - r * (unsigned)R.P);
    } else {
        const int nk = a.n2 / kTile, di = q / R.P;
        i = tile / nk + di - 1;
        k = (tile % nk) * kTile - 1 + (q - di * R.P);
    }
    return i >= 0 && i < a.n0 && k >= 0 && k < a.n2;
}

// a row's accumulator (NOUT columns from col, this warp's lanes) to voxel v, if
// the position is one
template <int NOUT>
__device__ __forceinline__ void store_row(const ConvArgs& a, uint32_t col, int warp, long v, bool live, int ntot,
                                          int n0) {
#pragma unroll 1
    for (int c0 = 0; c0 < NOUT; c0 += 16) {
        float accv[16];
        tmem_ld16(col + ((uint32_t)(warp * 32) << 16) + (uint32_t)c0, accv);
        if (!live) continue;
        if (a.bias) {
#pragma unroll
            for (int q = 0; q < 16; ++q) accv[q] += a.bias[n0 + c0 + q];
        }
        if (a.relu) {
#pragma unroll
            for (int q = 0; q < 16; ++q) accv[q] = fmaxf(accv[q], 0.f);
        }
        if (a.mask) {
            const uint4* mp = reinterpret_cast<const uint4*>(a.mask + v * ntot + n0 + c0);
            uint4 mv[2] = {mp[0], mp[1]};
            const bf16* m = reinterpret_cast<const bf16*>(mv);
#pragma unroll
            for (int q = 0; q < 16; ++q)
                if (!(__bfloat162float(m[q]) > 0.f)) accv[q] = 0.f;
        }
        uint4 ov[2];
        __nv_bfloat162* o = reinterpret_cast<__nv_bfloat162*>(ov);
#pragma unroll
        for (int q = 0; q < 8; ++q) o[q] = __floats2bfloat162_rn(accv[2 * q], accv[2 * q + 1]);
        uint4* op = reinterpret_cast<uint4*>(a.out + v * ntot + n0 + c0);
        op[0] = ov[0];
        op[1] = ov[1];
    }
}

// this warp's 32 lanes of 16 consecutive columns to zero
__device__ __forceinline__ void tmem_zero16(uint32_t taddr) {
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1, %1, %1, %1, %1, %1, %1, %1, %1, %1, %1, %1, %1, %1, %1, %1};"
        ::"r"(taddr), "r"(0)
        : "memory");
}

// (two CTAs of nine warps put five on one scheduler: at most 96 registers, the
// bound for ten warps each; at 108 the second CTA stayed out, 840 -> 1445 us)
template <int CG, int NOUT, int JS, bool RING>
__global__ void __launch_bounds__(kRowThreads + 32, JS * NOUT <= 256 ? 2 : 1) k_conv_rows(ConvArgs a, RowPlan R) {
    using F = RowShape<CG, NOUT, JS>;
    constexpr int NQ = CG / 16;
    extern __shared__ __align__(1024) uint8_t smem[];
    const int NR = R.nr;
    const uint32_t chunk = (uint32_t)R.nvox * 16, set_bytes = (CG / 8) * chunk;
    uint64_t* full = reinterpret_cast<uint64_t*>(smem + NR * set_bytes + R.nw * F::WBYTES);
    uint64_t* empty = full + kRowRing;
    uint64_t* wfull = empty + kRowRing;   // [2]
    uint64_t* wempty = wfull + 2;   // [2]
    uint64_t* tfull = wempty + 2;   // [JS]
    uint64_t* tempty = tfull + JS;  // [JS]
    uint64_t* fin = tempty + JS;    // every MMA of the CTA has completed
    uint32_t* slot = reinterpret_cast<uint32_t*>(fin + 1);

    const int tid = threadIdx.x, warp = tid >> 5;
    const int n1 = a.n1, n2 = a.n2;
    const int seg = (int)blockIdx.x / R.tiles, tile = (int)blockIdx.x - seg * R.tiles;
    const int js = seg * R.rows, je = min(js + R.rows, n1);
    // input rows inside the grid (those outside are zero)
    const int jlo = max(js - 1, 0), jhi = min(je, n1 - 1);
    const int nqt = (a.in.c0 + a.in.c1) / 16, groups = nqt / NQ;

    if (tid == 0) {
        for (int r = 0; r < NR; ++r) {
            mbar_init(&full[r], kProducers);
            mbar_init(&empty[r], 1);
        }
        for (int q = 0; q < 2; ++q) {
            mbar_init(&wfull[q], kProducers);
            mbar_init(&wempty[q], 1);
        }
        for (int q = 0; q < JS; ++q) {
            mbar_init(&tfull[q], 1);
            mbar_init(&tempty[q], kProducers);
        }
        mbar_init(fin, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 8) tmem_alloc(slot, F::NCOLS);
    tc_before();
    __syncthreads();
    tc_after();
    const uint32_t tmem = *slot;
    if (warp < 4) {
#pragma unroll 1
        for (int c = 0; c < JS * NOUT; c += 16) tmem_zero16(tmem + ((uint32_t)(warp * 32) << 16) + (uint32_t)c);
        asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
    }
    tc_before();
    __syncthreads();
    tc_after();
    bool ok = true;
    const uint32_t base = smem_u32(smem), wb = base + NR * set_bytes;

    if (warp >= 4 && warp < 8) {
        // ---- loader: per group its weights, then its row-sets; the thread
        // fetches chunk h of positions q0, q0 + QS, ..., whose voxels (of row 0,
        // in either source; -1 outside the grid) it keeps
        constexpr int QS = kProducers * 8 / CG, M = (F::MAXVOX + QS - 1) / QS;
        const int lt = tid - 128, h = lt % (CG / 8), q0 = lt / (CG / 8);
        const int up = a.in.up0, c0 = a.in.c0;
        int v0[M], v1[M];
#pragma unroll
        for (int m = 0; m < M; ++m) {
            int i, k;
            const bool valid = row_voxel(a, R, tile, q0 + m * QS, i, k);
            v0[m] = valid ? (i >> up) * (n1 >> up) * (n2 >> up) + (k >> up) : -1;
            v1[m] = valid ? i * n1 * n2 + k : -1;
        }
        int e = 0;  // row-sets so far
        for (int g = 0; ok && g < groups; ++g) {
            if (!mbar_wait(&wempty[g & 1], ((uint32_t)(g >> 1) & 1) ^ 1)) {
                ok = false;
                break;
            }
            // packed blocks (tap, kc channels), of their 16-byte pieces (8
            // outputs, 8 channels, output) those of 16 channels, to
            // ((di, dk), u, dj = 2, 1, 0)
            constexpr int WCH = NOUT * 32 / 16;  // pieces of 16 channels
            const int lk = R.lk, nb = (nqt * 2) >> lk;
            for (int c = lt; c < 27 * NQ * WCH; c += kProducers) {
                const int blk = c / WCH, t = blk / NQ, u = blk - t * NQ;
                const int di = t / 9, dj = (t / 3) % 3, dk = t % 3;
                const int w = (int)blockIdx.y * WCH + (c - blk * WCH), ch8 = (g * NQ + u) * 2 + ((w >> 3) & 1);
                const int at = ((((w >> 4) << lk) + (ch8 & ((1 << lk) - 1))) << 3) + (w & 7);
                cp16(wb + (g & 1) * F::WBYTES + ((((di * 3 + dk) * NQ + u) * 3 + 2 - dj) * WCH + (c - blk * WCH)) * 16,
                     a.wpack + (((long)(t * nb + (ch8 >> lk)) * R.ntot << lk) + at) * 8, true);
            }
            cp_arrive(&wfull[g & 1]);
            const int ch = g * CG + h * 8;
            const bool first = ch < c0;
            for (int jj = jlo; jj <= jhi; ++jj, ++e) {
                const int r = e % NR;
                if (!mbar_wait(&empty[r], ((uint32_t)(e / NR) & 1) ^ 1)) {
                    ok = false;
                    break;
                }
                const bf16* p = first ? a.in.src0 + (long)(jj >> up) * (n2 >> up) * c0 + ch
                                      : a.in.src1 + (long)jj * n2 * a.in.c1 + (ch - c0);
                const int cs = first ? c0 : a.in.c1;
                const uint32_t d = base + r * set_bytes + h * chunk + q0 * 16;
#pragma unroll
                for (int m = 0; m < M; ++m) {
                    const int v = first ? v0[m] : v1[m];
                    if (q0 + m * QS < R.nvox) cp16(d + m * QS * 16, v >= 0 ? p + (long)v * cs : a.wpack, v >= 0);
                }
                cp_arrive(&full[r]);
            }
        }
    } else if (tid == 256) {
        // ---- MMA issue
        int e = 0;
        for (int g = 0; ok && g < groups; ++g) {
            if (!mbar_wait(&wfull[g & 1], (uint32_t)(g >> 1) & 1)) ok = false;
            const uint32_t wg = wb + (g & 1) * F::WBYTES;
            for (int jj = jlo; ok && jj <= jhi; ++jj, ++e) {
                if (!mbar_wait(&full[e % NR], (uint32_t)(e / NR) & 1)) {
                    ok = false;
                    break;
                }
                asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
                tc_after();
                // output rows lo .. hi of jj-1 .. jj+1 lie in the segment
                const int lo = max(js, jj - 1), hi = min(je - 1, jj + 1);
                // RING: a row beyond the JS-th takes the accumulator of the JS-th before it
                if (RING && hi == jj + 1 && hi - js >= JS) {
                    if (!mbar_wait(&tempty[(hi - js) % JS], (uint32_t)((hi - js) / JS - 1) & 1)) {
                        ok = false;
                        break;
                    }
                    tc_after();
                }
                const uint32_t set = base + (e % NR) * set_bytes;
                auto issue = [&](int row, int at, int n) {
                    const uint32_t idesc = idesc_bf16(kTile, n * NOUT, false, false);
                    const uint32_t d = tmem + (uint32_t)(at * NOUT), wj = wg + (uint32_t)((row - (jj - 1)) * NOUT * 32);
#pragma unroll
                    for (int di = 0; di < 3; ++di) {
#pragma unroll
                        for (int dk = 0; dk < 3; ++dk) {
#pragma unroll
                            for (int u = 0; u < NQ; ++u)
                                umma(d, sdesc(set + 2 * u * chunk + (di * R.P + dk) * 16, chunk, 128),
                                     sdesc(wj + (uint32_t)(((di * 3 + dk) * NQ + u) * 3 * NOUT * 32), 128, 256), idesc, 1u);
                        }
                    }
                };
                if constexpr (RING) {
                    // one MMA, or two where the accumulators begin again
#pragma unroll 1
                    for (int row = lo, n; row <= hi; row += n) {
                        const int at = (row - js) % JS;
                        n = min(hi - row + 1, JS - at);
                        issue(row, at, n);
                    }
                } else {
                    issue(lo, lo - js, hi - lo + 1);
                }
                umma_commit(&empty[e % NR]);
                if (g == groups - 1) {
                    // complete: the row before, and at the end the last one
                    if (jj - 1 >= js) umma_commit(&tfull[RING ? (jj - 1 - js) % JS : jj - 1 - js]);
                    if (jj == jhi && jj < je) umma_commit(&tfull[RING ? (jj - js) % JS : jj - js]);
                }
            }
            if (ok) umma_commit(&wempty[g & 1]);
        }
        umma_commit(fin);
    }

    if (warp < 4) {
        // ---- epilogue: position tid of the tile, one row and one voxel into
        // the run
        int i, k;
        const bool live = row_voxel(a, R, tile, R.P + 1 + tid, i, k);
        for (int j = js; j < je; ++j) {
            const int at = RING ? (j - js) % JS : j - js;
            bool done = mbar_wait(&tfull[at], RING ? (uint32_t)((j - js) / JS) & 1 : 0u);
            done = __all_sync(0xffffffffu, done);
            if (!done) {
                ok = false;
                break;
            }
            tc_after();
            store_row<NOUT>(a, tmem + (uint32_t)(at * NOUT), warp, ((long)i * n1 + j) * n2 + k, live, R.ntot,
                            (int)blockIdx.y * NOUT);
            if (RING && j + JS < je) {  // the accumulator's next row
#pragma unroll 1
                for (int c = 0; c < NOUT; c += 16)
                    tmem_zero16(tmem + ((uint32_t)(warp * 32) << 16) + (uint32_t)(at * NOUT + c));
                asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
                tc_before();
                asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(&tempty[at])) : "memory");
            }
        }
    }

    if (!ok && a.err) atomicExch(a.err, kErrTimeout);
    tc_before();
    __syncthreads();
    if (warp == 8) {
        tc_after();
        mbar_wait(fin, 0);  // no MMA may still write the accumulators
        tmem_free(tmem, F::NCOLS);
    }
}

constexpr int conv_stages(int kc, int nout) {
    return (96 * 1024) / (kc * 2 * (kTile + nout)) > 6   ? 6
           : (96 * 1024) / (kc * 2 * (kTile + nout)) < 2 ? 2
                                                          : (96 * 1024) / (kc * 2 * (kTile + nout));
}

template <int KC, int NOUT>
cudaError_t conv_inst(const ConvArgs& a, cudaStream_t s) {
    constexpr int S = conv_stages(KC, NOUT);
    constexpr int smem = S * (KC * 2 * (kTile + NOUT)) + (2 * S + 1) * 8 + 16;
    cudaError_t e = cudaFuncSetAttribute(k_conv<KC, NOUT, S>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    if (e != cudaSuccess) return e;
    const long V = (long)a.n0 * a.n1 * a.n2;
    k_conv<KC, NOUT, S><<<(unsigned)((V + kTile - 1) / kTile), kThreads, smem, s>>>(a);
    return cudaGetLastError();
}

template <int NOUT>
cudaError_t wgrad_inst(const WgradArgs& a, cudaStream_t s) {
    constexpr int S = 3;
    constexpr int smem = S * (128 * kTile * 2 + NOUT * kTile * 2) + (2 * S + 1) * 8 + 16;
    cudaError_t e = cudaFuncSetAttribute(k_wgrad<NOUT, S>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    if (e != cudaSuccess) return e;
    k_wgrad<NOUT, S><<<dim3((unsigned)(a.rows_pad / 128), (unsigned)a.nsplit), kThreads, smem, s>>>(a);
    return cudaGetLastError();
}

template <int COUT>
cudaError_t wgrad_rows(const WgradArgs& a, cudaStream_t s) {
    constexpr int smem = WgRowShape<COUT>::smem;
    cudaError_t e = cudaFuncSetAttribute(k_wgrad_rows<COUT>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    if (e != cudaSuccess) return e;
    k_wgrad_rows<COUT><<<dim3((unsigned)a.nsplit, 3, (unsigned)((a.in.c0 + a.in.c1) / 16)), kThreads, smem, s>>>(a);
    return cudaGetLastError();
}

// the plan's extents of a run, and rows of a ring in `bytes` of shared memory
template <int CG, int NOUT, int JS>
int rows_ring(const ConvArgs& a, RowPlan& R, int bytes) {
    R.stream = a.n2 % kTile != 0;
    R.P = R.stream ? a.n2 + 1 : kTile + 2;
    R.nvox = 2 * R.P + kTile + 2;
    R.nw = std::min(2, (a.in.c0 + a.in.c1) / CG);
    const int fixed = R.nw * RowShape<CG, NOUT, JS>::WBYTES + RowShape<CG, NOUT, JS>::BARS;
    return std::min(kRowRing, (bytes - fixed) / ((CG / 8) * R.nvox * 16));
}
constexpr int kRowsTwo = 113 * 1024, kRowsOne = 227 * 1024;  // shared memory of a CTA, two and one an SM

template <int CG, int NOUT, int JS, bool RING>
cudaError_t rows_go(const ConvArgs& a, const RowPlan& R, int parts, cudaStream_t s) {
    using F = RowShape<CG, NOUT, JS>;
    const int smem = R.nr * (CG / 8) * R.nvox * 16 + R.nw * F::WBYTES + F::BARS;
    const auto kernel = k_conv_rows<CG, NOUT, JS, RING>;
    cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    if (e != cudaSuccess) return e;
    const unsigned segs = (unsigned)((a.n1 + R.rows - 1) / R.rows);
    kernel<<<dim3((unsigned)R.tiles * segs, (unsigned)parts), kRowThreads, smem, s>>>(a, R);
    return cudaGetLastError();
}

template <int CG, int NOUT, int JS>
cudaError_t rows_inst(const ConvArgs& a, int kc, int parts, cudaStream_t s) {
    using F = RowShape<CG, NOUT, JS>;
    RowPlan R;
    R.lk = kc == 64 ? 3 : kc == 32 ? 2 : 1;
    R.ntot = NOUT * parts;
    // as deep a ring as fits: two CTAs an SM where their accumulators do
    R.nr = rows_ring<CG, NOUT, JS>(a, R, F::NCOLS == 256 ? kRowsTwo : kRowsOne);
    const bool two = F::NCOLS == 256 && R.nr >= 2;
    if (R.nr < 2) R.nr = rows_ring<CG, NOUT, JS>(a, R, kRowsOne);
    if (R.nr < 1) return cudaErrorInvalidValue;
    const long tiles = R.stream ? ((long)a.n0 * R.P + kTile - 1) / kTile : (long)a.n0 * (a.n2 / kTile);
    R.tiles = (int)tiles;
    // Rows a CTA, at the least cost, the most rows where that is equal: input rows
    // walked (two more than it owns) times the CTAs an SM gets.  With one group of
    // channels a row is complete after its three input rows and its accumulator can
    // go to the JS-th row after it, so a CTA may take more rows; its start and end
    // take about as long as 5 rows, and two CTAs on an SM slow each other to 1.4
    // times a row's time (64^3, 16 -> 32: 18.7 us with 8 rows a CTA, 23.0 with 16).
    // 16 -> 48 at 128^3 takes 113 us with up to 32 rows, 155 with 5.  With one CTA an
    // SM that was slower (32 -> 32 at 128^3 202 us against 189).
    const bool march = two && R.nw == 1;
    long best = 0;
    for (int t = std::min(march ? kRowsMost : JS, a.n1); t >= 1; --t) {
        const long ctas = tiles * parts * ((a.n1 + t - 1) / t);
        const long cost = !march         ? (ctas + kSms - 1) / kSms * (t + 2)
                          : ctas <= kSms ? 5 * (t + 2 + 5)
                                         : (ctas + 2 * kSms - 1) / (2 * kSms) * (7 * (t + 2) + 25);
        if (!best || cost < best) {
            best = cost;
            R.rows = t;
        }
    }
    if constexpr (F::NCOLS == 256) {
        if (R.rows > JS) return rows_go<CG, NOUT, JS, true>(a, R, parts, s);
    }
    return rows_go<CG, NOUT, JS, false>(a, R, parts, s);
}

}  // namespace

// The row-marching kernel covers 16 to 64 output channels, or 96 and 128 in
// halves (32 -> 96 at 64^3: 146 -> 89 us, 64 -> 128 at 32^3: 53 -> 28), from
// inputs in whole blocks of 16: it was the faster one at every level of the
// network (figures at the kernel).  Rows are whole 128-voxel segments or have at
// most 256 voxels: a longer run would not leave room for the weights, nor the
// loader's registers; those use k_conv.  So do more than 256 input channels,
// which no layer has and the tests of this kernel do not reach (it would be the
// faster one there too: 320 -> 16 at 64^3 236 us against 1397).
bool rows_supported(int cin, int nout, int n2) {
    const bool out = nout == 16 || nout == 32 || nout == 48 || nout == 64 || nout == 96 || nout == 128;
    return out && cin % 16 == 0 && cin <= 256 && (n2 % kTile == 0 || n2 <= 256);
}

// 48 output channels, parts of them: 5 rows a CTA where two CTAs fit an SM, else 10
cudaError_t rows48(const ConvArgs& a, int kc, int parts, cudaStream_t s) {
    RowPlan R;
    return rows_ring<16, 48, 5>(a, R, kRowsTwo) >= 2 ? rows_inst<16, 48, 5>(a, kc, parts, s)
                                                     : rows_inst<16, 48, 10>(a, kc, parts, s);
}

// Rows a CTA: 16 of 16 output channels, 8 of 32 and 5 of 48 (256 columns of
// tensor memory each: two CTAs an SM, one's start and end under the other's
// rows), 8 of 64, and of 32 from groups of 32 input channels 16 (all of it).  With
// one CTA an SM, 16 rows of 32 and 10 of 48, 48 -> 32 at 128^3 took 316 us (now 272)
// and 32 -> 48 306 (246), 32 -> 96 at 64^3 86 (64); a tap an MMA 16 -> 32 132 (103)
// and 16 -> 48 133 (113).
// 10 rows of 48 stay where the weights leave two CTAs no ring: 32 -> 48 on
// 40 x 24 x 200 40 us against 47.  Groups of 32 input channels where both weight
// buffers leave room for a ring.
cudaError_t rows_launch(const ConvArgs& a, int kc, int nout, cudaStream_t s) {
    const int cin = a.in.c0 + a.in.c1;
    if (nout == 16) return rows_inst<16, 16, 16>(a, kc, 1, s);
    if (nout == 32) return cin % 32 || (a.n2 % kTile && a.n2 > kTile) ? rows_inst<16, 32, 8>(a, kc, 1, s)
                                                                     : rows_inst<32, 32, 16>(a, kc, 1, s);
    if (nout == 48) return rows48(a, kc, 1, s);
    if (nout == 64) return rows_inst<16, 64, 8>(a, kc, 1, s);
    if (nout == 96) return rows48(a, kc, 2, s);
    if (nout == 128) return rows_inst<16, 64, 8>(a, kc, 2, s);
    return cudaErrorInvalidValue;
}

bool conv_supported(int kc, int nout) {
    switch (kc) {
        case 16: return nout == 16 || nout == 32 || nout == 48 || nout == 64;
        case 32: return nout == 16 || nout == 32 || nout == 64 || nout == 96;
        case 64: return nout == 32 || nout == 64 || nout == 128;
        default: return false;
    }
}

bool wgrad_supported(int cout) { return cout == 16 || cout == 32 || cout == 64; }

#define BUN_CONV_CASE(KC, N) \
    if (kc == KC && nout == N) return conv_inst<KC, N>(a, s);

cudaError_t conv_launch(const ConvArgs& a, int kc, int nout, cudaStream_t s) {
    // 16-channel weight blocks, and the widest outputs: the row-marching kernel
    if ((kc == 16 || nout >= 96) && a.in.c0 % 16 == 0 && a.in.c1 % 16 == 0 &&
        rows_supported(a.in.c0 + a.in.c1, nout, a.n2))
        return rows_launch(a, kc, nout, s);
    BUN_CONV_CASE(16, 16)
    BUN_CONV_CASE(16, 32)
    BUN_CONV_CASE(16, 48)
    BUN_CONV_CASE(16, 64)
    BUN_CONV_CASE(32, 16)
    BUN_CONV_CASE(32, 32)
    BUN_CONV_CASE(32, 64)
    BUN_CONV_CASE(32, 96)
    BUN_CONV_CASE(64, 32)
    BUN_CONV_CASE(64, 64)
    BUN_CONV_CASE(64, 128)
    return cudaErrorInvalidValue;
}
#undef BUN_CONV_CASE

cudaError_t wgrad_launch(const WgradArgs& a, int cout, cudaStream_t s) {
    // rows in whole steps of 16 voxels (an MMA's K) and channels in whole blocks
    // of 16; a row's 8 channels must come from one source
    const int cin = a.in.c0 + a.in.c1;
    // and blocks of rows that are filled: a block's MMAs are those of W =
    // 128 / cout rows, whatever it holds.  Below 24 whole voxel columns of it the
    // gather was faster or equal (64 x 1 x 128, 16 -> 16: 14.7 against 20.8 us;
    // 128 x 2 x 32 14.6 against 20.8), above it the rows (128 x 4 x 128, 39.2
    // against 31.0), unless the grid has W rows (128 x 16 x 16, 29.0 against 27.0)
    const bool filled = a.n1 * cout >= 128 || (long)a.n1 * std::min(a.n2, kWgVox) * cout >= 24 * 128;
    if (filled && a.n2 % 16 == 0 && cin % 16 == 0 && a.in.c0 % 8 == 0) {
        if (cout == 16) return wgrad_rows<16>(a, s);
        if (cout == 32) return wgrad_rows<32>(a, s);
        if (cout == 64) return wgrad_rows<64>(a, s);
    }
    if (cout == 16) return wgrad_inst<16>(a, s);
    if (cout == 32) return wgrad_inst<32>(a, s);
    if (cout == 64) return wgrad_inst<64>(a, s);
    return cudaErrorInvalidValue;
}

}  // namespace bun
