// bfft_internal.h -- structures, register DFTs and launchers shared by the
// kernels of the FFT Poisson solver (bfft.cu, bfft_pair.cu, bfft_tri.cu).
#pragma once

#include <cuda_runtime.h>

namespace bfft {

// boundary pair of an axis (FourierTransforms.C:130-226)
enum Pair { P_EMPTY = 0, P_DD = 1, P_NN = 2, P_DN = 3, P_ND = 4, P_CC = 5 };
// output of a transform: halfcomplex of Z, Re(Z), Re(post Z), -Im(post Z)
enum Mode { M_R2HC = 0, M_HC2R = 1, M_RE = 2, M_NEG_IM = 3 };

constexpr int kThreads = 256;
constexpr int kMaxN = 512;

// lines along one axis: line l starts at (l / inner) * outer + (l % inner) * inner_stride
struct Lines {
    int n;             // cells along the axis
    long stride;       // element stride along the axis
    long inner;        // lines per outer index
    long inner_stride;
    long outer_stride;
    long count;
    int line_fast;     // consecutive lines are adjacent in memory (strided axes)
};

struct Transform {
    int M, logM, mode;
    int kind;             // Kind
    int odd;              // K_DCT2 / K_DCT3: the sine kinds RODFT10 / RODFT01
    int logN;             // log2 of the line length (transformed extents are powers of two)
    int logLB;            // log2 of the lines per CTA
    const double2* pre;   // n entries, nullptr: 1
    const double2* post;  // n entries, nullptr: 1
    const double2* tw;    // M entries: exp(-2 pi i q / M)
};

struct Tri {
    int ns, cyclic;
    double shift;
    double s0;            // first diagonal entry of a pinned (singular) mode
    int pin;              // the solve direction is N-N or periodic: the mode whose two
                          // eigenvalues are zero is singular and pinned (tridiagonalSolver.C)
    const double* A;      // D_k = ((e - A_k) - B_k)
    const double* B;
    const double* DU;
    const double* DL;
    const double* ev1;    // eigenvalue / h^2 of the first transform direction
    const double* ev2;
    int dir1_inner;       // the first transform direction is the inner line coordinate
    // modes with equal eigenvalues share one factorisation: class of each
    // inner / outer line coordinate, a representative coordinate per class
    const int* clsI;
    const int* clsO;
    const int* repI;
    const int* repO;
    int nci, nco;
    double* mfac;         // [ns][modes]: DL_k / Dh_{k-1} (k_tri_apply only)
    double* rfac;         // [ns][modes]: 1 / Dh_k
};

constexpr int kTriAhead = 8;  // rows a tridiagonal sweep loads ahead
constexpr int kSplitBlocks = 592;  // partial maxima of the face coefficients

struct Prep {
    int n0, n1, n2;
    double shift, scale;
    double corr[6];       // face terms subtracted on the boundary cells of each face
};

// the prep of the first transform's input: -b - shift x_old - face terms,
// times 1/normalisation (FFTPoissonSolver.C:116-183)
struct LoadPrep {
    int on;
    int axis;             // the transform axis
    int n1, n2;
    const double* xo;     // nullptr: no ddt term
    Prep P;
};

__device__ __forceinline__ long line_base(const Lines& L, long l) {
    // along axes 0 and 2 the outer stride is inner * inner_stride: no division
    if (L.outer_stride == L.inner * L.inner_stride) return l * L.inner_stride;
    const unsigned lu = (unsigned)l, in = (unsigned)L.inner;  // line counts fit 32 bits
    const unsigned o = lu / in;
    return (long)o * L.outer_stride + (long)(lu - o * in) * L.inner_stride;
}

__device__ __forceinline__ double2 cmul(double2 a, double2 b) {
    return make_double2(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x);
}

// cos and sin of a pi / 8, a = 0..7: the twiddles of the register DFTs (R <= 16)
__host__ __device__ constexpr double cos8(int a) {
    return a == 0   ? 1.0
           : a == 1 ? 0.92387953251128675613
           : a == 2 ? 0.70710678118654752440
           : a == 3 ? 0.38268343236508977173
           : a == 4 ? 0.0
           : a == 5 ? -0.38268343236508977173
           : a == 6 ? -0.70710678118654752440
                    : -0.92387953251128675613;
}
__host__ __device__ constexpr double sin8(int a) { return a <= 4 ? cos8(4 - a) : cos8(a - 4); }

__host__ __device__ constexpr int brev_c(int i, int logR) {
    int r = 0;
    for (int b = 0; b < logR; ++b) r |= ((i >> b) & 1) << (logR - 1 - b);
    return r;
}

// x * exp(-i pi p / h) for compile-time p < h <= 8
template <int P, int H>
__device__ __forceinline__ double2 rot(double2 x) {
    constexpr int a = P * (8 / H);
    if constexpr (a == 0) {
        return x;
    } else if constexpr (a == 4) {
        return make_double2(x.y, -x.x);
    } else {
        constexpr double c = cos8(a), sn = sin8(a);
        return make_double2(x.x * c + x.y * sn, x.y * c - x.x * sn);
    }
}

template <int H, int I, int P, int R>
__device__ __forceinline__ void bfly(double2 (&v)[R]) {
    const double2 u = v[I + P];
    const double2 t = rot<P, H>(v[I + P + H]);
    v[I + P] = make_double2(u.x + t.x, u.y + t.y);
    v[I + P + H] = make_double2(u.x - t.x, u.y - t.y);
}

template <int H, int I, int P, int R>
__device__ __forceinline__ void bfly_group(double2 (&v)[R]) {
    if constexpr (P < H) {
        bfly<H, I, P, R>(v);
        bfly_group<H, I, P + 1, R>(v);
    }
}

template <int H, int I, int R>
__device__ __forceinline__ void bfly_stage(double2 (&v)[R]) {
    if constexpr (I < R) {
        bfly_group<H, I, 0, R>(v);
        bfly_stage<H, I + 2 * H, R>(v);
    }
}

template <int H, int R>
__device__ __forceinline__ void bfly_stages(double2 (&v)[R]) {
    if constexpr (H < R) {
        bfly_stage<H, 0, R>(v);
        bfly_stages<2 * H, R>(v);
    }
}

// in-register DFT of R points (natural order in and out): bit reversal,
// then radix-2 stages with the exact twiddles of kCos8 / kSin8
template <int R, int LOGR>
__device__ __forceinline__ void dft_regs(double2 (&v)[R]) {
    double2 t[R];
#pragma unroll
    for (int i = 0; i < R; ++i) t[i] = v[brev_c(i, LOGR)];
#pragma unroll
    for (int i = 0; i < R; ++i) v[i] = t[i];
    bfly_stages<1, R>(v);
}

__device__ __forceinline__ void cp8(void* smem, const void* gmem, bool valid) {
    const unsigned sa = (unsigned)__cvta_generic_to_shared(smem);
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;\n" ::"r"(sa), "l"(gmem), "r"(valid ? 8 : 0)
                 : "memory");
}
// 16 bytes, of which `bytes` (0, 8 or 16) are read and the rest zero-filled
__device__ __forceinline__ void cp16(void* smem, const void* gmem, int bytes) {
    const unsigned sa = (unsigned)__cvta_generic_to_shared(smem);
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(sa), "l"(gmem), "r"(bytes) : "memory");
}
__device__ __forceinline__ void cp_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
__device__ __forceinline__ void cp_wait_all() { asm volatile("cp.async.wait_group 0;\n" ::: "memory"); }

// Transform kinds.  K_TRIG: one zero-padded M = 2N point complex FFT per
// line with a pre-twiddle of the input and a post-twiddle of the output
// (the quarter-wave kinds REDFT11 / RODFT11).  The others put two real lines
// into one N-point complex FFT (line 2u as the real part, line 2u + 1 as the
// imaginary part) and separate the two spectra afterwards from
// Z(k) and conj Z(N - k):
//   K_R2HC  forward real FFT, halfcomplex output
//   K_HC2R  inverse real FFT of halfcomplex input (unnormalised)
//   K_DCT2  REDFT10 by Makhoul's reordering (J. Makhoul, "A fast cosine
//           transform in one and two dimensions", IEEE TASSP 28 (1980)):
//           v = (x0, x2, x4, ..., x5, x3, x1), X_k = 2 Re(e^{-i pi k/2N} V_k);
//           with `odd`, RODFT10 as REDFT10 of (-1)^n x_n, read backwards
//   K_DCT3  REDFT01, the inverse of that reordering: V_k = e^{i pi k/2N}
//           (X_k - i X_{N-k}) (X_N = 0), v = IDFT(V), x_2n = v_n,
//           x_2n+1 = v_{N-1-n}; with `odd`, RODFT01 as (-1)^n REDFT01 of
//           the reversed input
// so every kind the solver meets on a periodic, Dirichlet-Dirichlet or
// Neumann-Neumann axis costs half an N-point complex FFT per line.
enum Kind { K_R2HC = 0, K_HC2R = 1, K_TRIG = 2, K_DCT2 = 3, K_DCT3 = 4 };

// the paired kinds on lines of 32 to 512 points (bfft_pair.cu)
constexpr int kPairMinLog = 5;
constexpr int kPairMaxLog = 9;
cudaError_t launch_pair(const double* in, double* out, const Lines& L, const Transform& T, const LoadPrep& LP,
                        bool adjacent, cudaStream_t st);

// the tridiagonal solves with a line shared by many threads (bfft_tri.cu);
// lines of a CTA for this many rows and lines, 0: too long
int tri_tile_lines(int ns, long count, int sms);
cudaError_t launch_tri_factor(const Tri& T, cudaStream_t st);
cudaError_t launch_tri_chunks(double* w, const Lines& L, const Tri& T, int tl, cudaStream_t st);

}  // namespace bfft
