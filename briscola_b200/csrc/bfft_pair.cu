// bfft_pair.cu -- the paired transforms (two real lines in one N-point
// complex FFT: real Fourier, cosine and sine kinds, bfft_internal.h) on lines
// of 32 to 512 points.
//
// A pass over the field reads and writes 16 B per complex point, and through
// shared memory it can afford only a few more such moves before those bound
// it.  So the lines go straight from memory into the registers of the first
// radix-16 pass, 16 independent loads a thread; the inverse kinds also store
// straight from the last pass's registers, and the forward kinds separate the
// two lines' spectra from one shared-memory copy, each pair of frequencies
// (k, N - k) read once.  2048 complex points a CTA, 128 threads of 16 points
// each, four CTAs an SM (128 registers): one CTA's loads run under the
// others' arithmetic, with no staging buffer.
//
// Consecutive threads take consecutive line pairs along the strided axes and
// consecutive points along k, so every load and store is a run of whole
// sectors.
//
// Measured, 256^3, us a pass (268 MB, 41 us at the copy rate), against the
// persistent kernel with a cp.async staging buffer that it replaces
// (k_transform, 12 warps an SM; it keeps the short lines and the quarter-wave
// kinds): real forward along k 123 -> 47, strided 128 -> 55, inverse along k
// 112 -> 48, strided 130 -> 51.

#include "bfft_internal.h"

#include <cstdint>

namespace bfft {

namespace {

constexpr int kPairThreads = 128;
constexpr int kPairPoints = 2048;  // complex points of a tile
constexpr int kPairSlots = kPairPoints + kPairPoints / 8;

// tile index -> shared-memory slot (16 B): one pad slot after every 16 and
// one after every line, so that the first pass's writes (stride 16) and the
// same point of consecutive lines fall in different bank groups
template <int LOGN>
__device__ __forceinline__ int slot(int i) {
    return i + (i >> 4) + (i >> LOGN);
}

// the point whose value sits at position p of Makhoul's order (even points
// first, then the odd ones backwards)
template <int N>
__device__ __forceinline__ int unmakhoul(int p) {
    return p < N / 2 ? 2 * p : 2 * (N - 1 - p) + 1;
}

// group g of a pass with 2^LOGG groups a line -> (line pair u, group j)
template <int LOGG, int LOGLB, bool LF>
__device__ __forceinline__ void group_of(int g, int& u, int& j) {
    if constexpr (LF) {
        u = g & ((1 << LOGLB) - 1);
        j = g >> LOGLB;
    } else {
        u = g >> LOGG;
        j = g & ((1 << LOGG) - 1);
    }
}

// the passes after the first (LOGNS points of a line done so far): radix 16
// while 16 or more remain; the last one hands each result to store(u, k, z)
template <int LOGN, int LOGNS, int LOGLB, bool LF, typename Store>
__device__ __forceinline__ void pair_passes(double2* __restrict__ buf, const double2* __restrict__ tw, Store&& store) {
    constexpr int LOGR = LOGN - LOGNS >= 4 ? 4 : LOGN - LOGNS;
    constexpr int R = 1 << LOGR, G = 16 / R, LOGG = LOGN - LOGR;
    constexpr bool last = LOGNS + LOGR == LOGN;
    double2 v[G][R];
#pragma unroll
    for (int gi = 0; gi < G; ++gi) {
        int u, j;
        group_of<LOGG, LOGLB, LF>((int)threadIdx.x + gi * kPairThreads, u, j);
#pragma unroll
        for (int r = 0; r < R; ++r) v[gi][r] = buf[slot<LOGN>((u << LOGN) + j + (r << LOGG))];
        const int step = (j & ((1 << LOGNS) - 1)) << (LOGN - LOGNS - LOGR);
#pragma unroll
        for (int r = 1; r < R; ++r) v[gi][r] = cmul(v[gi][r], __ldg(tw + r * step));
        dft_regs<R, LOGR>(v[gi]);
    }
    if constexpr (last) {
        store.begin();
#pragma unroll
        for (int gi = 0; gi < G; ++gi) {
            int u, j;
            group_of<LOGG, LOGLB, LF>((int)threadIdx.x + gi * kPairThreads, u, j);
#pragma unroll
            for (int r = 0; r < R; ++r) store(u, j + (r << LOGNS), v[gi][r]);
        }
    } else {
        __syncthreads();
#pragma unroll
        for (int gi = 0; gi < G; ++gi) {
            int u, j;
            group_of<LOGG, LOGLB, LF>((int)threadIdx.x + gi * kPairThreads, u, j);
            const int at = (u << LOGN) + ((j >> LOGNS) << (LOGNS + LOGR)) + (j & ((1 << LOGNS) - 1));
#pragma unroll
            for (int r = 0; r < R; ++r) buf[slot<LOGN>(at + (r << LOGNS))] = v[gi][r];
        }
        __syncthreads();
        pair_passes<LOGN, LOGNS + LOGR, LOGLB, LF>(buf, tw, store);
    }
}

// one line pair of the tile: its element offsets and which lines exist
struct PairLine {
    long a, b;
    bool va, vb;
};

// forward kinds: the spectrum stays in shared memory for the separation
template <int LOGN>
struct KeepSpectrum {
    double2* buf;
    __device__ __forceinline__ void begin() const { __syncthreads(); }
    __device__ __forceinline__ void operator()(int u, int k, double2 z) const { buf[slot<LOGN>((u << LOGN) + k)] = z; }
};

// inverse kinds: point q of both lines, straight to memory
template <int LOGN, int KIND, bool LF>
struct StorePoints {
    double* out;
    const Lines* L;
    long tile;
    PairLine own;  // strided axes: a thread's line pair is the same in every pass
    int odd, adjacent;
    __device__ __forceinline__ void begin() const {}
    __device__ __forceinline__ void operator()(int u, int k, double2 z) const;
};

template <int LOGN, bool LF>
__device__ __forceinline__ PairLine pair_line(const Lines& L, long tile, int u) {
    constexpr int LBC = kPairPoints >> LOGN;
    const long la = tile * (2 * LBC) + 2 * u;
    PairLine P;
    P.va = la < L.count;
    P.vb = la + 1 < L.count;
    if constexpr (LF) {
        P.a = P.va ? line_base(L, la) : 0;
        P.b = P.vb ? line_base(L, la + 1) : 0;
    } else {
        P.a = la << LOGN;  // axis-2 lines are consecutive rows
        P.b = (la + 1) << LOGN;
    }
    return P;
}

template <bool LF>
__device__ __forceinline__ void put2(double* out, const PairLine& P, long off, int adjacent, double a, double b) {
    if (LF && adjacent && P.vb) {
        *reinterpret_cast<double2*>(out + P.a + off) = make_double2(a, b);
    } else {
        if (P.va) out[P.a + off] = a;
        if (P.vb) out[P.b + off] = b;
    }
}

template <int LOGN, int KIND, bool LF>
__device__ __forceinline__ void StorePoints<LOGN, KIND, LF>::operator()(int u, int k, double2 z) const {
    constexpr int N = 1 << LOGN;
    const int q = KIND == K_DCT3 ? unmakhoul<N>(k) : k;
    // the forward FFT of conj(A + i B) is conj(a + i b)
    double a = z.x, b = -z.y;
    if (KIND == K_DCT3 && odd && (q & 1)) {
        a = -a;
        b = -b;
    }
    put2<LF>(out, LF ? own : pair_line<LOGN, LF>(*L, tile, u), LF ? (long)q * L->stride : q, adjacent, a, b);
}

template <int LOGN, int KIND, bool LF>
__global__ void __launch_bounds__(kPairThreads, 4) k_pair(const double* in, double* out, const __grid_constant__ Lines L,
                                                          Transform T, const __grid_constant__ LoadPrep LP,
                                                          int adjacent) {
    extern __shared__ __align__(16) double2 buf[];
    constexpr int N = 1 << LOGN, S = N / 16;
    constexpr int LOGLB = 11 - LOGN;  // line pairs of a tile
    constexpr int LBC = 1 << LOGLB;
    constexpr bool SPEC = KIND == K_HC2R || KIND == K_DCT3;  // spectral input
    const long tile = blockIdx.x;
    int u, j;
    group_of<LOGN - 4, LOGLB, LF>((int)threadIdx.x, u, j);
    const PairLine P = pair_line<LOGN, LF>(L, tile, u);

    // position p = j + r N/16 of the transform's order -> point of the line
    auto point = [&](int p) {
        if constexpr (KIND == K_DCT2) return unmakhoul<N>(p);
        if constexpr (KIND == K_DCT3) return T.odd ? N - 1 - p : p;
        return p;
    };
    double2 v[16];
#pragma unroll
    for (int r = 0; r < 16; ++r) {
        const long off = LF ? (long)point(j + r * S) * L.stride : point(j + r * S);
        if (LF && adjacent && P.vb) {
            v[r] = *reinterpret_cast<const double2*>(in + P.a + off);
        } else {
            v[r].x = P.va ? in[P.a + off] : 0.0;
            v[r].y = P.vb ? in[P.b + off] : 0.0;
        }
    }
    if (LP.on) {
        // the first transform forms the right-hand side: -b - shift x_old -
        // face terms, times 1/normalisation
        auto fixed_terms = [&](long l) {
            const unsigned in_ = (unsigned)L.inner;
            const long co = (unsigned)l / in_, ci = (unsigned)l - (unsigned)co * in_;
            const int a0 = LP.axis == 0 ? 1 : 0, a1 = LP.axis == 2 ? 1 : 2;
            const int e0 = a0 == 0 ? LP.P.n0 : LP.P.n1, e1 = a1 == 1 ? LP.P.n1 : LP.P.n2;
            double f = 0.0;
            if (co == 0) f += LP.P.corr[2 * a0];
            if (co == e0 - 1) f += LP.P.corr[2 * a0 + 1];
            if (ci == 0) f += LP.P.corr[2 * a1];
            if (ci == e1 - 1) f += LP.P.corr[2 * a1 + 1];
            return f;
        };
        const long la = tile * (2 * LBC) + 2 * u;
        const double fa = P.va ? fixed_terms(la) : 0.0, fb = P.vb ? fixed_terms(la + 1) : 0.0;
#pragma unroll
        for (int r = 0; r < 16; ++r) {
            const int q = point(j + r * S);
            const long off = LF ? (long)q * L.stride : q;
            double a = -v[r].x, b = -v[r].y;
            if (LP.xo) {
                if (P.va) a -= LP.P.shift * LP.xo[P.a + off];
                if (P.vb) b -= LP.P.shift * LP.xo[P.b + off];
            }
            double ta = fa, tb = fb;
            if (q == 0) {
                ta += LP.P.corr[2 * LP.axis];
                tb += LP.P.corr[2 * LP.axis];
            }
            if (q == N - 1) {
                ta += LP.P.corr[2 * LP.axis + 1];
                tb += LP.P.corr[2 * LP.axis + 1];
            }
            v[r] = make_double2(P.va ? (a - ta) * LP.P.scale : 0.0, P.vb ? (b - tb) * LP.P.scale : 0.0);
        }
    }
    if constexpr (KIND == K_DCT2) {
        if (T.odd) {  // the odd points, positions N/2 .. N-1, change sign
#pragma unroll
            for (int r = 8; r < 16; ++r) v[r] = make_double2(-v[r].x, -v[r].y);
        }
    }
    if constexpr (SPEC) {
        // frequency k = j + r N/16 needs the values at k and N - k
#pragma unroll
        for (int r = 0; r < 16; ++r) buf[slot<LOGN>((u << LOGN) + j + r * S)] = v[r];
        __syncthreads();
#pragma unroll
        for (int r = 0; r < 16; ++r) {
            const int k = j + r * S;
            const double2 h = v[r];
            const double2 g = buf[slot<LOGN>((u << LOGN) + ((N - k) & (N - 1)))];
            double ar, ai, br, bi;
            if constexpr (KIND == K_HC2R) {
                // A_k = (r_k, i_k) of a halfcomplex line, i_k stored at N - k
                const bool lo = 2 * k <= N, real = k == 0 || 2 * k == N;
                ar = lo ? h.x : g.x;
                br = lo ? h.y : g.y;
                ai = real ? 0.0 : lo ? g.x : -h.x;
                bi = real ? 0.0 : lo ? g.y : -h.y;
            } else {
                // V_k = c_k (X_k - i X_{N-k}), c_k = e^{i pi k / 2N}, X_N = 0
                const double2 c = __ldg(T.pre + k);
                const double gx = k ? g.x : 0.0, gy = k ? g.y : 0.0;
                ar = c.x * h.x + c.y * gx;
                ai = c.y * h.x - c.x * gx;
                br = c.x * h.y + c.y * gy;
                bi = c.y * h.y - c.x * gy;
            }
            v[r] = make_double2(ar - bi, -(ai + br));  // conj(A + i B)
        }
        __syncthreads();
    }
    dft_regs<16, 4>(v);
#pragma unroll
    for (int r = 0; r < 16; ++r) buf[slot<LOGN>((u << LOGN) + 16 * j + r)] = v[r];
    __syncthreads();
    if constexpr (SPEC) {
        pair_passes<LOGN, 4, LOGLB, LF>(buf, T.tw, StorePoints<LOGN, KIND, LF>{out, &L, tile, P, T.odd, adjacent});
    } else {
        pair_passes<LOGN, 4, LOGLB, LF>(buf, T.tw, KeepSpectrum<LOGN>{buf});
        __syncthreads();
        // frequencies k and N - k of both lines from Z(k) and Z(N - k); k = 0
        // goes with N / 2
        constexpr int LOGH = LOGN - 1;
#pragma unroll 4
        for (int s = 0; s < kPairPoints / 2 / kPairThreads; ++s) {
            int uu, k;
            group_of<LOGH, LOGLB, LF>((int)threadIdx.x + s * kPairThreads, uu, k);
            const int k2 = k ? N - k : N / 2;
            const double2 z = buf[slot<LOGN>((uu << LOGN) + k)], y = buf[slot<LOGN>((uu << LOGN) + k2)];
            const PairLine Q = LF ? P : pair_line<LOGN, LF>(L, tile, uu);
            double a1, b1, a2, b2;
            int q1 = k, q2 = k2;
            if constexpr (KIND == K_R2HC) {
                // A = (Z_k + conj Z_{N-k}) / 2, B = (Z_k - conj Z_{N-k}) / 2i:
                // the real parts at k, the imaginary parts at N - k
                a1 = k ? 0.5 * (z.x + y.x) : z.x;
                b1 = k ? 0.5 * (z.y + y.y) : z.y;
                a2 = k ? 0.5 * (z.y - y.y) : y.x;
                b2 = k ? -0.5 * (z.x - y.x) : y.y;
            } else {
                // 2 Re(w_k A_k) and 2 Re(w_k B_k), w_k = e^{-i pi k / 2N}
                const double2 w1 = __ldg(T.post + k), w2 = __ldg(T.post + k2);
                const double2 y1 = k ? y : z, z2 = k ? z : y;  // Z(N - k) of each frequency
                a1 = w1.x * (z.x + y1.x) - w1.y * (z.y - y1.y);
                b1 = w1.x * (z.y + y1.y) + w1.y * (z.x - y1.x);
                a2 = w2.x * (y.x + z2.x) - w2.y * (y.y - z2.y);
                b2 = w2.x * (y.y + z2.y) + w2.y * (y.x - z2.x);
                if (T.odd) {
                    q1 = N - 1 - q1;
                    q2 = N - 1 - q2;
                }
            }
            put2<LF>(out, Q, LF ? (long)q1 * L.stride : q1, adjacent, a1, b1);
            put2<LF>(out, Q, LF ? (long)q2 * L.stride : q2, adjacent, a2, b2);
        }
    }
}

template <int KIND, bool LF, int LOGN>
cudaError_t launch_one(int logN, const double* in, double* out, const Lines& L, const Transform& T, const LoadPrep& LP,
                       int adjacent, cudaStream_t st) {
    if constexpr (LOGN <= kPairMaxLog) {
        if (logN != LOGN) return launch_one<KIND, LF, LOGN + 1>(logN, in, out, L, T, LP, adjacent, st);
        constexpr int lines = 2 * (kPairPoints >> LOGN);
        const long tiles = (L.count + lines - 1) / lines;
        k_pair<LOGN, KIND, LF><<<(unsigned)tiles, kPairThreads, kPairSlots * sizeof(double2), st>>>(in, out, L, T, LP,
                                                                                                 adjacent);
        return cudaGetLastError();
    } else {
        return cudaErrorInvalidValue;
    }
}

template <bool LF>
cudaError_t launch_kinds(const double* in, double* out, const Lines& L, const Transform& T, const LoadPrep& LP,
                         int adjacent, cudaStream_t st) {
    switch (T.kind) {
        case K_R2HC: return launch_one<K_R2HC, LF, kPairMinLog>(T.logN, in, out, L, T, LP, adjacent, st);
        case K_HC2R: return launch_one<K_HC2R, LF, kPairMinLog>(T.logN, in, out, L, T, LP, adjacent, st);
        case K_DCT2: return launch_one<K_DCT2, LF, kPairMinLog>(T.logN, in, out, L, T, LP, adjacent, st);
        case K_DCT3: return launch_one<K_DCT3, LF, kPairMinLog>(T.logN, in, out, L, T, LP, adjacent, st);
        default: return cudaErrorInvalidValue;
    }
}

}  // namespace

// adjacent: consecutive lines of a pair are neighbours in memory (strided
// axes with an even number of cells along k); then, and where both arrays
// start on 16 bytes, the two move as one vector
cudaError_t launch_pair(const double* in, double* out, const Lines& L, const Transform& T, const LoadPrep& LP,
                        bool adjacent, cudaStream_t st) {
    const bool aligned = ((reinterpret_cast<uintptr_t>(in) | reinterpret_cast<uintptr_t>(out)) & 15) == 0;
    const int adj = adjacent && aligned;
    return L.line_fast ? launch_kinds<true>(in, out, L, T, LP, adj, st) : launch_kinds<false>(in, out, L, T, LP, adj, st);
}

}  // namespace bfft
