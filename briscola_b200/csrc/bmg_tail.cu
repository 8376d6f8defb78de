// bmg_tail.cu -- the coarse end of a V or F cycle in one thread-block
// cluster, with every level it visits held in the cluster's shared memory.
//
// On the small levels a pass is a few thousand cells: a launch per pass
// costs its latency and not its work.  Here the right-hand side of the first
// level is read once, every smoothing pass, transfer and coarse solve of the
// sub-cycle runs out of shared memory with a barrier between them, and the
// first level's x is written once.  The sequence of steps (MG.C:19-130, V or
// F cycle) comes from the host as a list.
//
// What bounds it: the number of dependent passes times the latency of one
// (shared loads, a chain of multiply-adds, the barrier), and on the
// larger levels the shared-memory bandwidth of one SM (13 loads an update).
// So levels above kTailGather cells are spread over the CTAs of the cluster,
// whole i-planes each, one cell update per thread and pass; a CTA pushes the
// values of its outer planes into its neighbours' halo planes as it computes
// them, and the cluster's hardware barrier ends the pass.  Smaller levels
// run on CTA 0 alone, where __syncthreads is the cheaper barrier.
//
// Measured (solves, one B200; before: one 512-thread CTA passing over levels
// of at most 4096 cells in L2, V cycles only): 16^3 cavity FP64 724 -> 404 us,
// 64^3 cavity FP64 1430 -> 900 us, 96 x 192 x 24 F cycles FP64 5300 -> 2670 us
// (with the whole loop in the kernel, where level 0 fits: 16^3 313 us).
// A pass of an 8^3 level takes about 700 cycles on CTA 0, one of 32^3 over
// 16 CTAs 2000, half of it the barrier and the halo stores it waits for; a
// launch per pass costs 5000.
//
// Rows are parity-split in shared memory ([k = -1][even k][odd k][k = n2],
// whatever n2 is), so a colour pass reads and writes consecutive words.  Per
// cell the arithmetic and its order are those of the per-pass kernels
// (gs_value, restrict_quad_item / k_residual_restrict, prolong_quad_item /
// k_prolong_correct, coarse_solve_block).  gs_value is shared and rounds
// explicitly; the transfers are written out here again, and that the compiler
// contracts both copies alike is a tested property: whole solves are
// bit-identical (tests/test_gpu_tail.py, tests/test_gpu_cluster_tail.py).

#include <cooperative_groups.h>

#include "bmg_grid.cuh"
#include "bmg_stencil.cuh"

namespace bmg {

namespace cg = cooperative_groups;

namespace {

// q = a / d for a < 2^16 and d < 2^16: m = ceil(2^32 / d), m = 0 for d = 1
__device__ __forceinline__ int div_by(int a, unsigned m) { return m ? (int)__umulhi((unsigned)a, m) : a; }

// position of logical k (-1 .. n2) in a shared-memory row
template <typename T>
__device__ __forceinline__ int spos(const TailLevel<T>& L, int k) {
    return (k >= 0 && k < L.n2) ? (k & 1) * L.ne + (k >> 1) : k;
}

// this CTA's planes of a level: first plane and how many
struct Own {
    int p0, cnt;
};
template <typename T>
__device__ __forceinline__ Own own_planes(const TailLevel<T>& L, int rank) {
    const Planes p = tail_own(L.n0, L.P, rank);
    return {p.first, p.count};
}

// stores x of cell (i, j, k) at word c (local plane li of cnt), its periodic
// images in its own plane, and its copies in the halo planes of the CTAs
// that own planes i - 1 and i + 1
template <typename T>
__device__ __forceinline__ void tail_store(const TailLevel<T>& L, T* sm, int rank, int cnt, int li, int i, int j,
                                           int k, int c, T v) {
    T* x = sm + L.x;
    x[c] = v;
    if (L.per1) {
        if (j == 0) x[c + L.n1 * L.sj] = v;
        if (j == L.n1 - 1) x[c - L.n1 * L.sj] = v;
    }
    if (L.per2) {
        const int c0 = c - spos(L, k);
        if (k == 0) x[c0 + L.n2] = v;
        if (k == L.n2 - 1) x[c0 - 1] = v;
    }
    if (li == 0 && (i > 0 || L.per0)) {
        const int up = i > 0 ? i - 1 : L.n0 - 1;  // its upper halo plane
        const int t = div_by(up, L.mP), slot = min(L.P, L.n0 - t * L.P) + 1;
        T* d = x + c + (slot - 1) * L.si;
        if (t != rank) d = cg::this_cluster().map_shared_rank(d, t);
        *d = v;
    }
    if (li == cnt - 1 && (i < L.n0 - 1 || L.per0)) {
        const int dn = i < L.n0 - 1 ? i + 1 : 0;  // its lower halo plane
        const int t = div_by(dn, L.mP);
        T* d = x + c - cnt * L.si;
        if (t != rank) d = cg::this_cluster().map_shared_rank(d, t);
        *d = v;
    }
}

// couplings of cell (i, j, k) (bmg_stencil.cuh: couplings) from shared
// memory; li: local plane
template <typename T, bool VAR>
__device__ __forceinline__ void tail_couplings(const TailLevel<T>& L, const T* sm, int li, int i, int j, int k,
                                               T w[6]) {
    const T* t = sm + L.tab;
    w[0] = t[i];
    w[1] = t[L.n0 + i];
    t += 2 * L.n0;
    w[2] = t[j];
    w[3] = t[L.n1 + j];
    t += 2 * L.n1;
    w[4] = t[k];
    w[5] = t[L.n2 + k];
    if (VAR) {
        const T* l0 = sm + L.lam[0] + (li * L.n1 + j) * L.n2 + k;
        const T* l1 = sm + L.lam[1] + (li * (L.n1 + 1) + j) * L.n2 + k;
        const T* l2 = sm + L.lam[2] + (li * L.n1 + j) * (L.n2 + 1) + k;
        w[0] *= l0[0];
        w[1] *= l0[L.n1 * L.n2];
        w[2] *= l1[0];
        w[3] *= l1[L.n2];
        w[4] *= l2[0];
        w[5] *= l2[1];
    }
}

// byte address of a word of this CTA's shared memory in CTA t's
template <typename T>
__device__ __forceinline__ unsigned word_at(const T* p, int t) {
    unsigned a = (unsigned)__cvta_generic_to_shared(p), r;
    asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(t));
    return r;
}
__device__ __forceinline__ void st_cluster(unsigned a, float v) {
    asm volatile("st.shared::cluster.f32 [%0], %1;" ::"r"(a), "f"(v) : "memory");
}
__device__ __forceinline__ void st_cluster(unsigned a, double v) {
    asm volatile("st.shared::cluster.f64 [%0], %1;" ::"r"(a), "d"(v) : "memory");
}

// ends a step: the cluster's barrier where its CTAs share the level, this
// CTA's otherwise
__device__ __forceinline__ void step_end(bool all) {
    if (all) {
        asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
        asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
    } else {
        __syncthreads();
    }
}

// One cell of a thread for a whole smoothing step: addresses (words from the
// level's x), its periodic images' distances (0: none) and what gs_value takes.
template <typename T, bool VAR>
struct TailCell {
    int c, cm, cp, imj, imk;
    T wk[2], wij[VAR ? 4 : 1], b, inv;
};

// A smoothing step: n red-black colour passes over this CTA's planes of a
// level, the colours alternating from `first`.  A thread owns one pair of
// neighbouring cells along k, one of each colour, for the whole step: their
// couplings, right-hand sides and addresses are set up once, so a pass is six
// loads, the update, and the stores.
template <typename T, bool VAR>
__device__ __forceinline__ void tail_smooth(const TailLevel<T>& D, T* sm, int rank, int first, int n) {
    const bool all = D.dist;
    const int ne = D.ne, n1 = D.n1, n2 = D.n2, si = D.si, sj = D.sj;
    const int it = threadIdx.x;
    T* x = sm + D.x;
    TailCell<T, VAR> A{}, B{};  // of the first and of the second pass's colour
    T wij[4] = {T(0), T(0), T(0), T(0)};
    bool haveA = false, haveB = false;
    // bit 0, 1: a copy goes to the owner of plane i-1 (i+1), from this address on
    unsigned push = 0, up = 0, dn = 0;
    {
        const Own o = own_planes(D, rank);
        if (it < o.cnt * n1 * ne) {
            const int ij = div_by(it, D.mne), m = it - ij * ne;
            const int li = div_by(ij, D.mn1), j = ij - li * n1, i = o.p0 + li;
            const int row = (li + 1) * si + (j + 1) * sj + 1;
            if (li == 0 && (i > 0 || D.per0)) {
                push |= 1u;
                const int t = div_by(i > 0 ? i - 1 : D.n0 - 1, D.mP);
                up = word_at(x + min(D.P, D.n0 - t * D.P) * si, t);
            }
            if (li == o.cnt - 1 && (i < D.n0 - 1 || D.per0)) {
                push |= 2u;
                dn = word_at(x, div_by(i < D.n0 - 1 ? i + 1 : 0, D.mP)) - (unsigned)(o.cnt * si * sizeof(T));
            }
            auto fill = [&](TailCell<T, VAR>& C, int colour) {
                const int h = (colour ^ (i + j + D.cpar)) & 1, k = 2 * m + h;
                if (k >= n2) return false;
                C.c = row + h * ne + m;
                C.cm = row + (h ? m : (m > 0 ? ne + m - 1 : -1));
                C.cp = row + (h ? (m + 1 < ne ? m + 1 : n2) : ne + m);
                C.imj = !D.per1 ? 0 : j == 0 ? n1 * sj : j == n1 - 1 ? -n1 * sj : 0;
                // k = 0 is the row's first word, its image n2 words on; k =
                // n2-1's image is the word before the row
                C.imk = !D.per2 ? 0 : k == 0 ? n2 : k == n2 - 1 ? row - 1 - C.c : 0;
                C.b = sm[D.b + ij * n2 + h * ne + m];
                T w[6];
                tail_couplings<T, VAR>(D, sm, li, i, j, k, w);
                C.inv = gs_inv(w);
                C.wk[0] = w[4];
                C.wk[1] = w[5];
#pragma unroll
                for (int d = 0; d < 4; ++d) (VAR ? C.wij[d % (VAR ? 4 : 1)] : wij[d]) = w[d];
                return true;
            };
            haveA = fill(A, first);
            haveB = fill(B, 1 - first);
        }
    }
    auto pass = [&](const TailCell<T, VAR>& C, bool have) {
        if (have) {
            const T xn[6] = {x[C.c - si], x[C.c + si], x[C.c - sj], x[C.c + sj], x[C.cm], x[C.cp]};
            T w[6] = {wij[0], wij[1], wij[2], wij[3], C.wk[0], C.wk[1]};
            if (VAR) {
#pragma unroll
                for (int d = 0; d < 4; ++d) w[d] = C.wij[d % (VAR ? 4 : 1)];
            }
            const T v = gs_value(w, xn, C.b, C.inv);
            x[C.c] = v;
            if (push & 1u) st_cluster(up + C.c * (unsigned)sizeof(T), v);
            if (push & 2u) st_cluster(dn + C.c * (unsigned)sizeof(T), v);
            if (C.imj) x[C.c + C.imj] = v;
            if (C.imk) x[C.c + C.imk] = v;
        }
        step_end(all);
    };
#pragma unroll 1
    for (int e = 0; e < n; e += 2) {
        pass(A, haveA);
        if (e + 1 < n) pass(B, haveB);
    }
}

// b(q+1) = restriction of b(q) - A x(q) to the owner of each coarse plane,
// and x(q+1) = 0.  A CTA's fine planes come in whole pairs, so it forms the
// coarse planes over them.  Four lanes share a coarse cell, one fine row
// (a, e) each; the rows' shares are added in the order of the per-pass
// kernels.
template <typename T, bool VAR>
__device__ __forceinline__ void tail_restrict(const TailLevel<T>& F, const TailLevel<T>& C, T* sm, int rank) {
    const T* x = sm + F.x;
    const T* b = sm + F.b;
    const T* r0 = sm + F.ratio;
    const T* r1 = r0 + F.n0;
    const T* r2 = r1 + F.n1;
    const Own o = own_planes(F, rank);
    const int I0 = F.R0 == 2 ? o.p0 >> 1 : o.p0;
    const int cells = (F.R0 == 2 ? o.cnt >> 1 : o.cnt) * C.n1 * C.n2;
    const int lane = threadIdx.x & 31, sub = lane & 3, a = sub >> 1, e = sub & 1;
    for (int base = (int)threadIdx.x - lane; base < 4 * cells; base += kTailThreads) {
        const int item = (base + lane) >> 2;
        const bool ok = item < cells;
        const int cell = ok ? item : 0;
        const int IJ = div_by(cell, C.mn2), K = cell - IJ * C.n2;
        const int lI = div_by(IJ, C.mn1), J = IJ - lI * C.n1, I = I0 + lI;
        T rab = T(0), t0 = T(0), t1 = T(0), f0 = T(0), f1 = T(0);
        if (a < F.R0 && e < F.R1) {
            const int i = I * F.R0 + a, j = J * F.R1 + e, li = i - o.p0;
            rab = r0[i] * r1[j];
            const int row = (li + 1) * F.si + (j + 1) * F.sj + 1;
            const int brow = (li * F.n1 + j) * F.n2;
#pragma unroll
            for (int q = 0; q < 2; ++q) {
                if (q >= F.R2) break;
                const int k = K * F.R2 + q, pk = spos(F, k), c = row + pk;
                T w[6];
                tail_couplings<T, VAR>(F, sm, li, i, j, k, w);
                const T sv = w[0] * x[c - F.si] + w[1] * x[c + F.si] + w[2] * x[c - F.sj] + w[3] * x[c + F.sj] +
                             w[4] * x[row + spos(F, k - 1)] + w[5] * x[row + spos(F, k + 1)];
                const T d = w[0] + w[1] + w[2] + w[3] + w[4] + w[5];
                const T r = b[brow + pk] + d * x[c] - sv;
                if (q == 0) {
                    t0 = r;
                    f0 = r2[k];
                } else {
                    t1 = r;
                    f1 = r2[k];
                }
            }
        }
        T acc = T(0);
        if (F.quad) {
            const T t = f0 * t0 + f1 * t1;
#pragma unroll
            for (int s = 0; s < 4; ++s) {
                const T ra = __shfl_sync(0xffffffffu, rab, (lane & 28) + s);
                const T ts = __shfl_sync(0xffffffffu, t, (lane & 28) + s);
                acc += ra * ts;
            }
        } else {
            f0 = rab * f0;
            f1 = rab * f1;
#pragma unroll
            for (int s = 0; s < 4; ++s) {
                const T a0 = __shfl_sync(0xffffffffu, f0, (lane & 28) + s);
                const T b0 = __shfl_sync(0xffffffffu, t0, (lane & 28) + s);
                const T a1 = __shfl_sync(0xffffffffu, f1, (lane & 28) + s);
                const T b1 = __shfl_sync(0xffffffffu, t1, (lane & 28) + s);
                if ((s >> 1) < F.R0 && (s & 1) < F.R1) {
                    acc += a0 * b0;
                    if (F.R2 > 1) acc += a1 * b1;
                }
            }
        }
        if (ok && sub == 0) {
            const int t = div_by(I, C.mP);
            T* d = sm + C.b + ((I - t * C.P) * C.n1 + J) * C.n2 + spos(C, K);
            if (t != rank) d = cg::this_cluster().map_shared_rank(d, t);
            *d = acc;
        }
    }
    for (int c = threadIdx.x; c < C.xcells; c += kTailThreads) sm[C.x + c] = T(0);
}

// x(q) += prolongation of x(q+1).  The coarse planes that a CTA's fine planes
// need are copied to a scratch slab first where another CTA owns any of them.
template <typename T>
__device__ __forceinline__ void tail_prolong(const TailLevel<T>& F, const TailLevel<T>& C, T* sm, int rank,
                                             int scratch) {
    const Own o = own_planes(F, rank);
    const T* X = sm + C.x;
    const int first = F.R0 == 2 ? o.p0 >> 1 : o.p0;  // parent of the first own plane: slot 1 of X
    if (F.dist) {
        // slots 0 .. np + 1: planes first - 1 .. first + np (wrapped on a
        // periodic axis, a halo plane of the end CTA at a wall)
        const int np = F.R0 == 2 ? o.cnt >> 1 : o.cnt;
        const int words = o.cnt ? (np + 2) * C.si : 0;
        for (int e = threadIdx.x; e < words; e += kTailThreads) {
            const int s = e / C.si, p = e - s * C.si;
            int I = first - 1 + s;
            if (C.per0) I = I < 0 ? I + C.n0 : I >= C.n0 ? I - C.n0 : I;
            const int t = div_by(min(max(I, 0), C.n0 - 1), C.mP);
            const T* src = sm + C.x + (I - t * C.P + 1) * C.si + p;
            sm[scratch + e] = t == rank ? *src : *cg::this_cluster().map_shared_rank(src, t);
        }
        X = sm + scratch;
        __syncthreads();
    }
    const T* w0 = sm + F.pw;
    const int* pi = reinterpret_cast<const int*>(sm + F.pidx);
    const int cells = o.cnt * F.n1 * F.n2;
    for (int it = threadIdx.x; it < cells; it += kTailThreads) {
        const int ij = div_by(it, F.mn2), pos = it - ij * F.n2;
        const int li = div_by(ij, F.mn1), j = ij - li * F.n1, i = o.p0 + li;
        const int k = pos < F.ne ? 2 * pos : 2 * (pos - F.ne) + 1;
        const T wi = w0[i], wj = w0[F.n0 + j], wk = w0[F.n0 + F.n1 + k];
        const T ui = T(1) - wi, uj = T(1) - wj, uk = T(1) - wk;
        // the parent plane's slot, and that of the plane on the fine cell's side
        const int P = pi[2 * i], Q = pi[2 * i + 1];
        const int sP = P - first + 1, sQ = Q == P ? sP : sP + ((i & 1) ? 1 : -1);
        const int I0 = sP * C.si, I1 = sQ * C.si;
        const int* pj = pi + 2 * F.n0;
        const int J0 = (pj[2 * j] + 1) * C.sj, J1 = (pj[2 * j + 1] + 1) * C.sj;
        const int* pk = pj + 2 * F.n1;
        const int P0 = spos(C, pk[2 * k]) + 1, P1 = spos(C, pk[2 * k + 1]) + 1;
        const T v00 = uk * X[I0 + J0 + P0] + wk * X[I0 + J0 + P1];
        const T v01 = uk * X[I0 + J1 + P0] + wk * X[I0 + J1 + P1];
        const T v10 = uk * X[I1 + J0 + P0] + wk * X[I1 + J0 + P1];
        const T v11 = uk * X[I1 + J1 + P0] + wk * X[I1 + J1 + P1];
        const int c = (li + 1) * F.si + (j + 1) * F.sj + 1 + pos;
        T v = sm[F.x + c];
        v += ui * (uj * v00 + wj * v01) + wi * (uj * v10 + wj * v11);
        tail_store(F, sm, rank, o.cnt, li, i, j, k, c, v);
    }
}

// x = A^-1 b on the coarse solve level, one warp per row (coarse_solve_block).
// Spread: every CTA of the cluster takes rows, from CTA 0's b into CTA 0's x.
template <typename T>
__device__ __forceinline__ void tail_coarse(const TailLevel<T>& C, T* sm, double* sb, const double* __restrict__ ainv,
                                            int n, int rank, int nranks) {
    const T* b = sm + C.b;
    if (rank) b = cg::this_cluster().map_shared_rank(b, 0);
    for (int q = threadIdx.x; q < n; q += kTailThreads) {
        const int ij = div_by(q, C.mn2), k = q - ij * C.n2;
        sb[q] = (double)b[ij * C.n2 + spos(C, k)];
    }
    __syncthreads();
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    for (int r = warp * nranks + rank; r < n; r += kTailThreads / 32 * nranks) {
        double s = 0.0;
        for (int l = lane; l < n; l += 32) s += ainv[r * n + l] * sb[l];
        for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
        if (lane == 0) {
            const int ij = div_by(r, C.mn2), k = r - ij * C.n2;
            const int i = div_by(ij, C.mn1), j = ij - i * C.n1;
            const int c = (i + 1) * C.si + (j + 1) * C.sj + 1 + spos(C, k);
            T* sm0 = rank ? cg::this_cluster().map_shared_rank(sm, 0) : sm;
            tail_store(C, sm0, 0, C.n0, i, i, j, k, c, (T)s);
        }
    }
}

// ||b - A x||^2 of this CTA's planes of level 0 (unscaled: times the volumes),
// per cell as k_residual_norm; valid in thread 0
template <bool VAR>
__device__ __forceinline__ double tail_residual(const TailPlan<double>& P, const TailLevel<double>& L,
                                                const double* sm, int rank) {
    __shared__ double part[kTailThreads / 32];
    const double* x = sm + L.x;
    const Own o = own_planes(L, rank);
    const int cells = o.cnt * L.n1 * L.n2;
    double a = 0.0;
    for (int it = threadIdx.x; it < cells; it += kTailThreads) {
        const int ij = div_by(it, L.mn2), pos = it - ij * L.n2;
        const int li = div_by(ij, L.mn1), j = ij - li * L.n1, i = o.p0 + li;
        const int k = pos < L.ne ? 2 * pos : 2 * (pos - L.ne) + 1;
        const int row = (li + 1) * L.si + (j + 1) * L.sj + 1, c = row + pos;
        double w[6];
        tail_couplings<double, VAR>(L, sm, li, i, j, k, w);
        const double xn[6] = {x[c - L.si], x[c + L.si], x[c - L.sj], x[c + L.sj], x[row + spos(L, k - 1)],
                              x[row + spos(L, k + 1)]};
        const double r = res_value(w, xn, x[c], sm[L.b + ij * L.n2 + pos]);
        const double V = __ldg(P.g.tab64 + P.g.to.h[0] + i) * __ldg(P.g.tab64 + P.g.to.h[1] + j) *
                         __ldg(P.g.tab64 + P.g.to.h[2] + k);
        a += (V * r) * (V * r);
    }
    for (int s = 16; s > 0; s >>= 1) a += __shfl_xor_sync(0xffffffffu, a, s);
    if ((threadIdx.x & 31) == 0) part[threadIdx.x >> 5] = a;
    __syncthreads();
    a = 0.0;
    if (threadIdx.x < 32) {
        a = part[threadIdx.x];
        for (int s = 16; s > 0; s >>= 1) a += __shfl_xor_sync(0xffffffffu, a, s);
    }
    return a;
}

// SOLVE (FP64, the first level is level 0): not one cycle but the solve's
// whole loop (MG.C:191-242), cycles until the residual decides, bounded by
// maxIter; a launch and its reload per cycle, the residual's and the
// decision's launches were half of a 16^3 solve's time.
template <typename T, bool VAR, bool SOLVE>
__global__ void __launch_bounds__(kTailThreads, 1) k_tail_cycle(const __grid_constant__ TailPlan<T> P) {
    extern __shared__ __align__(16) double smd[];
    double* sb = smd;  // ncoarse doubles, then the inverse where it fits
    double* ainv_s = smd + P.ncoarse + (P.ncoarse & 1);
    T* sm = reinterpret_cast<T*>(ainv_s + P.ainvWords);
    const int nranks = (int)cg::this_cluster().num_blocks(), rank = (int)cg::this_cluster().block_rank();
    // the level descriptors and the steps in shared memory: read with a
    // running index, the parameters miss the constant cache
    __shared__ TailLevel<T> lv[kMaxTail];
    __shared__ unsigned char ops[kMaxTailOps];
    for (int e = threadIdx.x; e < (int)(P.nlev * sizeof(TailLevel<T>) / 4); e += kTailThreads)
        reinterpret_cast<int*>(lv)[e] = reinterpret_cast<const int*>(P.v)[e];
    for (int e = threadIdx.x; e < P.nops; e += kTailThreads) ops[e] = P.ops[e];
    // what no earlier kernel of the solve writes (tables, face coefficients,
    // the coarse inverse) is on its way before the preceding grid is done
    for (int q = 0; q + 1 < P.nlev; ++q) {
        const TailLevel<T>& L = P.v[q];
        if (!L.dist && rank) break;
        const int n = L.n0 + L.n1 + L.n2;
        for (int e = threadIdx.x; e < n; e += kTailThreads) {
            const int d = e < L.n0 ? 0 : e < L.n0 + L.n1 ? 1 : 2;
            const int at = d == 0 ? e : d == 1 ? e - L.n0 : e - L.n0 - L.n1;
            const int nd = d == 0 ? L.n0 : d == 1 ? L.n1 : L.n2;
            T* t = sm + L.tab + 2 * (d == 0 ? 0 : d == 1 ? L.n0 : L.n0 + L.n1);
            t[at] = ldg(L.gtab + L.wl[d] + at);
            t[nd + at] = ldg(L.gtab + L.wh[d] + at);
            sm[L.ratio + e] = ldg(L.gratio + e);
            sm[L.pw + e] = ldg(L.gpw + e);
            int* pi = reinterpret_cast<int*>(sm + L.pidx);
            pi[2 * e] = __ldg(L.gpidx + 2 * e);
            pi[2 * e + 1] = __ldg(L.gpidx + 2 * e + 1);
        }
        if (VAR) {
            const Own o = own_planes(L, rank);
            for (int d = 0; d < 3; ++d) {
                const int f0 = o.cnt ? o.cnt + (d == 0) : 0, f1 = L.n1 + (d == 1), f2 = L.n2 + (d == 2);
                for (int e = threadIdx.x; e < f0 * f1 * f2; e += kTailThreads) {
                    const int ij = e / f2, k = e - ij * f2, li = ij / f1, j = ij - li * f1;
                    sm[L.lam[d] + e] = ldg(L.glam[d] + L.gbase + (o.p0 + li) * L.gsi + j * L.gsj +
                                           (L.gkh ? kpos_split(k, L.gkh) : k));
                }
            }
        }
    }
    const double* ainv = P.ainv;
    if (P.ainvWords && !rank) {
        for (int e = threadIdx.x; e < P.ncoarse * P.ncoarse; e += kTailThreads) ainv_s[e] = __ldg(P.ainv + e);
        ainv = ainv_s;
    }
    grid_dep_sync();
    {
        // the first level: b, and x with its ghosts (or zero)
        const TailLevel<T>& L = P.v[0];
        const Own o = own_planes(L, rank);
        for (int e = threadIdx.x; e < o.cnt * L.n1 * L.n2; e += kTailThreads) {
            const int ij = div_by(e, L.mn2), k = e - ij * L.n2, li = div_by(ij, L.mn1), j = ij - li * L.n1;
            sm[L.b + ij * L.n2 + spos(L, k)] =
                P.gb[L.gbase + (o.p0 + li) * L.gsi + j * L.gsj + (L.gkh ? kpos_split(k, L.gkh) : k)];
        }
        const Planes in = tail_read({o.p0, o.cnt});
        for (int e = threadIdx.x; e < L.xcells; e += kTailThreads) {
            T v = T(0);
            if (!P.zeroStart) {
                const int s = e / L.si, j = (e - s * L.si) / L.sj, p = e - s * L.si - j * L.sj - 1;
                const int k = p < 0 || p >= L.n2 ? p : p < L.ne ? 2 * p : 2 * (p - L.ne) + 1;
                if (s < in.count)
                    v = P.gx[L.gbase + (in.first + s) * L.gsi + (j - 1) * L.gsj + (L.gkh ? kpos_split(k, L.gkh) : k)];
            }
            sm[L.x + e] = v;
        }
    }
    // every CTA has started (its shared memory may be written) and is loaded
    step_end(nranks > 1);
    // the CTAs' shares of the norm and the decision, in CTA 0's and every
    // CTA's shared memory
    __shared__ double norms[kTailRanks];
    __shared__ int go;
    if (SOLVE && threadIdx.x == 0) go = P.st->keep_going;
    if (SOLVE) __syncthreads();
    while (!SOLVE || go) {
        for (int s = 0; s < P.nops; ++s) {
            const int op = ops[s] >> 3, q = ops[s] & 7;
            const TailLevel<T>& L = lv[q];
            const bool all = L.dist;  // every CTA takes part, and the cluster's barrier ends each pass
            if (op == TAIL_PRE || op == TAIL_POST) {
                if (all || !rank)
                    tail_smooth<T, VAR>(L, sm, rank, op == TAIL_PRE ? L.pre : L.post, op == TAIL_PRE ? L.npre : L.npost);
            } else if (op == TAIL_RESTRICT) {
                if (!all && rank) continue;
                tail_restrict<T, VAR>(L, lv[q + 1], sm, rank);
                step_end(all);
            } else if (op == TAIL_PROLONG) {
                if (!all && rank) continue;
                // the coarse level is complete (CTA 0 may have worked alone on it)
                if (all && !lv[q + 1].dist) step_end(true);
                tail_prolong<T>(L, lv[q + 1], sm, rank, P.scratch);
                step_end(all);
            } else if (P.spread) {
                step_end(true);
                tail_coarse<T>(L, sm, sb, ainv, P.ncoarse, rank, nranks);
                step_end(true);
            } else if (!rank) {
                tail_coarse<T>(L, sm, sb, ainv, P.ncoarse, 0, 1);
                __syncthreads();
            }
        }
        if constexpr (SOLVE) {
            const double a = tail_residual<VAR>(P, lv[0], sm, rank);
            if (threadIdx.x == 0) st_cluster(word_at(norms + rank, 0), a);
            step_end(nranks > 1);
            if (!rank && threadIdx.x == 0) {
                double l2 = 0.0;
                for (int r = 0; r < nranks; ++r) l2 += norms[r];
                solve_decision(P.st, sqrt(l2), 1);
                for (int r = 0; r < nranks; ++r) {
                    const unsigned d = word_at(&go, r);
                    asm volatile("st.shared::cluster.s32 [%0], %1;" ::"r"(d), "r"(P.st->keep_going) : "memory");
                }
            }
            step_end(nranks > 1);
        } else {
            break;
        }
    }
    // x of the first level with its periodic images.  In a cluster of several
    // CTAs that level is spread, so the last step ended with the cluster's
    // barrier: no CTA touches another's shared memory any more
    const TailLevel<T>& L = P.v[0];
    const Own o = own_planes(L, rank);
    for (int e = threadIdx.x; e < o.cnt * L.n1 * L.n2; e += kTailThreads) {
        const int ij = div_by(e, L.mn2), p = e - ij * L.n2, li = div_by(ij, L.mn1), j = ij - li * L.n1;
        const int k = p < L.ne ? 2 * p : 2 * (p - L.ne) + 1;
        const T v = sm[L.x + (li + 1) * L.si + (j + 1) * L.sj + 1 + p];
        store_x(P.g, P.g.base + (o.p0 + li) * P.g.si + j * P.g.sj + kpos(P.g, k), o.p0 + li, j, k, v);
    }
}

}  // namespace

template <typename T, bool VAR, bool SOLVE>
static cudaError_t launch_tail(const TailPlan<T>& P, cudaStream_t s) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(P.ranks);
    cfg.blockDim = dim3(kTailThreads);
    cfg.dynamicSmemBytes = P.smem;
    cfg.stream = s;
    cudaLaunchAttribute at[2];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = P.ranks;
    at[0].val.clusterDim.y = 1;
    at[0].val.clusterDim.z = 1;
    at[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = at;
    cfg.numAttrs = kProgrammaticLaunch ? 2 : 1;
    return cudaLaunchKernelEx(&cfg, k_tail_cycle<T, VAR, SOLVE>, P);
}

template <typename T, bool VAR>
cudaError_t launch_tail_cycle(const TailPlan<T>& P, cudaStream_t s) {
    return launch_tail<T, VAR, false>(P, s);
}

template <bool VAR>
cudaError_t launch_tail_solve(const TailPlan<double>& P, cudaStream_t s) {
    return launch_tail<double, VAR, true>(P, s);
}

template <typename T, bool VAR, bool SOLVE = false>
static int allow_tail() {
    const auto kernel = k_tail_cycle<T, VAR, SOLVE>;
    if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kTailSmem) != cudaSuccess) return 0;
    // a cluster lies in one GPC: a part of a device may hold a small one only,
    // or none
    const bool most = cudaFuncSetAttribute(kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) == cudaSuccess;
    for (int r = most ? kTailRanks : 8; r >= 1; r /= 2) {
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = dim3(r);
        cfg.blockDim = dim3(kTailThreads);
        cfg.dynamicSmemBytes = kTailSmem;
        cudaLaunchAttribute at;
        at.id = cudaLaunchAttributeClusterDimension;
        at.val.clusterDim.x = r;
        at.val.clusterDim.y = 1;
        at.val.clusterDim.z = 1;
        cfg.attrs = &at;
        cfg.numAttrs = 1;
        int n = 0;
        if (cudaOccupancyMaxActiveClusters(&n, kernel, &cfg) == cudaSuccess && n >= 1) return r;
    }
    return 0;
}

int configure_tail_kernels() {
    const int r = std::min({allow_tail<float, false>(), allow_tail<float, true>(), allow_tail<double, false>(),
                            allow_tail<double, true>(), allow_tail<double, false, true>(), allow_tail<double, true, true>()});
    if (r < kTailRanks) cudaGetLastError();  // a refused query is an answer
    return r;
}

template cudaError_t launch_tail_cycle<double, false>(const TailPlan<double>&, cudaStream_t);
template cudaError_t launch_tail_cycle<double, true>(const TailPlan<double>&, cudaStream_t);
template cudaError_t launch_tail_cycle<float, false>(const TailPlan<float>&, cudaStream_t);
template cudaError_t launch_tail_cycle<float, true>(const TailPlan<float>&, cudaStream_t);
template cudaError_t launch_tail_solve<false>(const TailPlan<double>&, cudaStream_t);
template cudaError_t launch_tail_solve<true>(const TailPlan<double>&, cudaStream_t);

}  // namespace bmg
