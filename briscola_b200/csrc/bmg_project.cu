// bmg_project.cu -- the steps either side of the pressure solve of a
// projection method, on the device, so that a time step keeps the velocity
// and the pressure in HBM (C ABI: bmg_project_rhs / bmg_project_correct in
// include/bmg.h).
//
// Right-hand side: the colocated divergence of the staggered velocity,
//   coloDiv(U)_c = sum over the cell's faces of U_f A_f (outward) / V_c
//   (divergenceScheme.C:116-150), divided by -C dt as the staggered solver
//   passes it (briscolaStaggered.C:92), or multiplied into the system form
//   b_sys = -V b of the linear solve (linearSystem.C:547-556).
// Correction: U_f -= C dt * stagReconstruct(flux)_f with the Poisson flux
//   lambda faceGrad(p) A (defaultPoissonSolver.C:110-123) and
//   stagReconstruct = -flux / A (exSchemesReconstruction.H:187-206): with the
//   outward face gradient (p_lo - p_c) delta, the face velocity loses
//   C dt lambda (p_c - p_lo) delta.  Zero-gradient walls leave their faces
//   unchanged; periodic faces wrap.
//
// Face arrays of axis d hold n_d + 1 faces along d (the face below cell q,
// then the top face), k fastest; on a periodic axis the last face is the
// first again and both are written.

#include "bmg_internal.h"

namespace bmg {

namespace {

// Both kernels stream the face arrays once, one cell (or face index) a
// thread over blocks of whole runs along k and several rows: memory bounds
// them, and on small bricks the number of CTAs does (a CTA of one row kept
// the 128 x 96 x 64 step's four launches at 10-14 us each).
__global__ void __launch_bounds__(256) k_project_rhs(const double* __restrict__ u0, const double* __restrict__ u1,
                                                     const double* __restrict__ u2, double* __restrict__ out,
                                                     ProjGeom G) {
    const int n1 = G.n[1], n2 = G.n[2];
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    const int j = blockIdx.y * blockDim.y + threadIdx.y;
    const int i = blockIdx.z;
    if (k >= n2 || j >= n1) return;
    const double h0 = G.h[0][i], h1 = G.h[1][j], h2 = G.h[2][k];
    const long f0 = ((long)i * n1 + j) * n2 + k;
    const long f1 = ((long)i * (n1 + 1) + j) * n2 + k;
    const long f2 = ((long)i * n1 + j) * (n2 + 1) + k;
    // sum of U A over the faces, then divided by V (A / V = 1 / h along each axis)
    const double div = (u0[f0 + (long)n1 * n2] - u0[f0]) / h0 + (u1[f1 + n2] - u1[f1]) / h1 +
                       (u2[f2 + 1] - u2[f2]) / h2;
    const double b = div / (-G.cdt);
    out[f0] = G.perVolume ? b : -(h0 * h1 * h2) * b;
}

// The three faces of index (i, j, k): those below cell (i, j, k) along each
// axis, and the top faces where i = n0, j = n1 or k = n2.  One pass: p is read
// once for the three axes.
__global__ void __launch_bounds__(256) k_project_correct(double* __restrict__ u0, double* __restrict__ u1,
                                                         double* __restrict__ u2, const double* __restrict__ p,
                                                         const double* __restrict__ lam0,
                                                         const double* __restrict__ lam1,
                                                         const double* __restrict__ lam2, ProjGeom G) {
    const int n0 = G.n[0], n1 = G.n[1], n2 = G.n[2];
    const int q[3] = {(int)blockIdx.z, (int)(blockIdx.y * blockDim.y + threadIdx.y),
                      (int)(blockIdx.x * blockDim.x + threadIdx.x)};
    const int i = q[0], j = q[1], k = q[2];
    if (j > n1 || k > n2) return;
    double* const us[3] = {u0, u1, u2};
    const double* const ls[3] = {lam0, lam1, lam2};
    const long st[3] = {(long)n1 * n2, n2, 1};
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        const int nA = G.n[a];
        if ((a != 0 && i == n0) || (a != 1 && j == n1) || (a != 2 && k == n2)) continue;
        const int e1 = a == 1 ? n1 + 1 : n1, e2 = a == 2 ? n2 + 1 : n2;
        int qc = q[a], ql = q[a] - 1;  // cells above and below the face
        if (qc == 0 || qc == nA) {
            if (!G.per[a]) continue;  // a wall: zero gradient
            qc = 0;  // across the periodic seam: the first and the last cell
            ql = nA - 1;
        }
        const double delta = 1.0 / (0.5 * (G.h[a][qc] + G.h[a][ql]));
        const long other = (a == 0 ? 0 : i * st[0]) + (a == 1 ? 0 : j * st[1]) + (a == 2 ? 0 : (long)k);
        const double g = (p[other + qc * st[a]] - p[other + ql * st[a]]) * delta;
        const long f = ((long)i * e1 + j) * e2 + k;
        const double l = ls[a] ? ls[a][f] : 1.0;
        us[a][f] -= G.cdt * (l * g);
    }
}

dim3 rows_block(int nk) { return nk > 32 ? dim3(64, 4) : dim3(32, 8); }

}  // namespace

void launch_project_rhs(const double* u0, const double* u1, const double* u2, double* out, const ProjGeom& G,
                        cudaStream_t s) {
    const dim3 b = rows_block(G.n[2]);
    k_project_rhs<<<dim3((G.n[2] + b.x - 1) / b.x, (G.n[1] + b.y - 1) / b.y, G.n[0]), b, 0, s>>>(u0, u1, u2, out, G);
}

void launch_project_correct(double* u0, double* u1, double* u2, const double* p, const double* lam0,
                            const double* lam1, const double* lam2, const ProjGeom& G, cudaStream_t s) {
    const dim3 b = rows_block(G.n[2] + 1);
    k_project_correct<<<dim3((G.n[2] + b.x) / b.x, (G.n[1] + b.y) / b.y, G.n[0] + 1), b, 0, s>>>(u0, u1, u2, p, lam0,
                                                                                            lam1, lam2, G);
}

}  // namespace bmg
