// bfft_tri.cu -- the tridiagonal solves of the FFT Poisson solver, each line
// shared by many threads.
//
// A mode's line of n rows is a serial elimination, and a dependent FP64
// multiply-add costs far more than its issue slot: one thread marching along
// 256 rows in memory (k_tri_apply, bfft.cu, which keeps the lines too long
// for this kernel) took 278 us for the 256^3 channel, and the same march out
// of shared memory, from both ends, 219 us.  With the factors 1 / D_k known,
// both sweeps are first-order recurrences, y_k = a_k - m_k y_{k-1}, so a line
// is cut into chunks of C rows, one thread each, held in registers: the chunk
// from a zero start and its product, a scan over the line's chunks for the
// value entering each (in shared memory, log2 steps), and the chunk again from
// that value.  The serial chain is 2 C rows and the scan instead of n, the field
// is read and written once, and a thread has all its 2 C loads in flight: 115 us
// there (139 with chunks of 16 rows, which also kept every row's product),
// 93 -> 12 us for 128 x 96 x 64 cells.
//
// Bound: memory (16 B a cell of the field and 8 B of each factor).

#include "bfft_internal.h"

#include <algorithm>

namespace bfft {

namespace {

constexpr int kTriMaxThreads = 512;

__device__ __forceinline__ double tri_diag(const Tri& T, int k, double e, bool singular) {
    const double d = (k == 0 && singular) ? T.s0 : (e - T.A[k]) - T.B[k];
    return d - T.shift;
}

// 1 / D_k of each class of modes, D_k = d_k - DL_k DU_{k-1} / D_{k-1}
// (tridiagonalSolver.C:343-353 without the right-hand side)
__global__ void k_tri_rfactor(Tri T) {
    const int mode = blockIdx.x * blockDim.x + threadIdx.x;
    const int modes = T.nci * T.nco;
    if (mode >= modes) return;
    const int ci = T.repI[mode % T.nci], co = T.repO[mode / T.nci];
    const int c1 = T.dir1_inner ? ci : co, c2 = T.dir1_inner ? co : ci;
    const double e1 = T.ev1[c1], e2 = T.ev2[c2];
    const double e = e1 + e2;
    const bool singular = T.pin && e1 == 0.0 && e2 == 0.0;
    double r = 1.0 / tri_diag(T, 0, e, singular);
    T.rfac[mode] = r;
    for (int k = 1; k < T.ns; ++k) {
        r = 1.0 / (tri_diag(T, k, e, singular) - T.DL[k] * r * T.DU[k - 1]);
        T.rfac[(long)k * modes + mode] = r;
    }
}

// the value entering this thread's chunk (q of Q, line t) from the chunks
// before it: chunk p maps y to a_p + b_p y.  Inclusive scan of the maps in
// shared memory, two buffers; the line starts from 0.
__device__ __forceinline__ double chunk_carry(double2* buf, int TL, int Q, int q, int t, double a, double b) {
    double2* cur = buf;
    double2* nxt = buf + TL * Q;
    cur[q * TL + t] = make_double2(a, b);
    __syncthreads();
    for (int d = 1; d < Q; d *= 2) {
        double2 m = cur[q * TL + t];
        if (q >= d) {
            const double2 l = cur[(q - d) * TL + t];
            m = make_double2(m.x + m.y * l.x, m.y * l.y);
        }
        nxt[q * TL + t] = m;
        __syncthreads();
        double2* s = cur;
        cur = nxt;
        nxt = s;
    }
    const double c = q ? cur[(q - 1) * TL + t].x : 0.0;
    __syncthreads();  // the buffers are free again
    return c;
}

// TL lines a CTA, Q chunks of C rows a line; thread (q, t), t fastest
template <int C>
__global__ void __launch_bounds__(kTriMaxThreads, C <= 8 ? 2 : 1)
    k_tri_chunks(double* __restrict__ w, const __grid_constant__ Lines L, const __grid_constant__ Tri T, int logTL,
                 int Q) {
    extern __shared__ __align__(16) double2 scan[];
    const int TL = 1 << logTL, t = threadIdx.x & (TL - 1), q = threadIdx.x >> logTL;
    const long l = (long)blockIdx.x * TL + t;
    const bool ok = l < L.count;
    const int k0 = q * C, modes = T.nci * T.nco;
    const unsigned inner = (unsigned)L.inner, lu = ok ? (unsigned)l : 0u;
    const int co = (int)(lu / inner), ci = (int)(lu - (unsigned)co * inner);
    const int rows = ok ? min(C, T.ns - k0) : 0;  // rows of this chunk
    const long st = L.stride;
    double* wl = w + line_base(L, lu) + k0 * st;
    const double* rl = T.rfac + T.clsO[co] * T.nci + T.clsI[ci] + (long)k0 * modes;
    double f[C], r[C];
    double rp = q && rows > 0 ? __ldg(rl - modes) : 0.0;  // 1 / D of the row before the chunk
    {
        const double* src = wl;
        const double* fac = rl;
#pragma unroll
        for (int e = 0; e < C; ++e) {
            f[e] = e < rows ? *src : 0.0;
            r[e] = e < rows ? __ldg(fac) : 0.0;
            src += st;
            fac += modes;
        }
    }
    // forward: y_k = f_k - (DL_k / D_{k-1}) y_{k-1}
    double m[C];
#pragma unroll
    for (int e = 0; e < C; ++e) {
        m[e] = e < rows && k0 + e > 0 ? -__ldg(T.DL + k0 + e) * rp : 0.0;
        rp = r[e];
    }
    double y = 0.0, b = 1.0;
#pragma unroll
    for (int e = 0; e < C; ++e) {
        y = f[e] + m[e] * y;
        b = m[e] * b;
    }
    y = chunk_carry(scan, TL, Q, q, t, y, b);
#pragma unroll
    for (int e = 0; e < C; ++e) {
        y = f[e] + m[e] * y;
        f[e] = y * r[e];
    }
    // backward: x_k = y_k / D_k - (DU_k / D_k) x_{k+1}
#pragma unroll
    for (int e = 0; e < C; ++e) m[e] = e < rows && k0 + e < T.ns - 1 ? -__ldg(T.DU + k0 + e) * r[e] : 0.0;
    double x = 0.0;
    b = 1.0;
#pragma unroll
    for (int e = C - 1; e >= 0; --e) {
        x = f[e] + m[e] * x;
        b = m[e] * b;
    }
    x = chunk_carry(scan, TL, Q, Q - 1 - q, t, x, b);
#pragma unroll
    for (int e = C - 1; e >= 0; --e) {
        x = f[e] + m[e] * x;
        f[e] = x;
    }
#pragma unroll
    for (int e = 0; e < C; ++e) {
        if (e < rows) *wl = f[e];
        wl += st;
    }
}

template <int C>
cudaError_t launch_c(double* w, const Lines& L, const Tri& T, int logTL, int Q, cudaStream_t st) {
    const int tl = 1 << logTL;
    k_tri_chunks<C><<<(unsigned)((L.count + tl - 1) / tl), tl * Q, (size_t)2 * tl * Q * sizeof(double2), st>>>(
        w, L, T, logTL, Q);
    return cudaGetLastError();
}

// rows of a chunk: as few as leave a CTA 16 lines (a whole 128-byte run of
// every row) within 512 threads
int chunk_rows(int ns) { return ns <= 64 ? 4 : ns <= 256 ? 8 : 16; }

}  // namespace

// Lines of a CTA: 16, halved while a line's chunks would not fit the CTA and
// (down to 4) while SMs would be left without one.  0: the line is too long
// (more than 2048 rows).
int tri_tile_lines(int ns, long count, int sms) {
    const int c = chunk_rows(ns), Q = (ns + c - 1) / c;
    int tl = 16;
    while (tl > 4 && tl * Q > kTriMaxThreads) tl /= 2;
    if (tl * Q > kTriMaxThreads) return 0;
    while (tl > 4 && count / tl < sms) tl /= 2;
    return tl;
}

cudaError_t launch_tri_factor(const Tri& T, cudaStream_t st) {
    const int modes = T.nci * T.nco;
    k_tri_rfactor<<<(modes + 127) / 128, 128, 0, st>>>(T);
    return cudaGetLastError();
}

cudaError_t launch_tri_chunks(double* w, const Lines& L, const Tri& T, int tl, cudaStream_t st) {
    const int c = chunk_rows(T.ns), Q = (T.ns + c - 1) / c;
    int logTL = 0;
    while ((1 << logTL) < tl) ++logTL;
    return c == 4   ? launch_c<4>(w, L, T, logTL, Q, st)
           : c == 8 ? launch_c<8>(w, L, T, logTL, Q, st)
                    : launch_c<16>(w, L, T, logTL, Q, st);
}

}  // namespace bfft
