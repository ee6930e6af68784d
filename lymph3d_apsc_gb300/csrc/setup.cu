// setup.cu -- device set-up kernels: geometry, polyhedron bounding boxes,
// operator block assembly, mass matrices and their Cholesky factors, RHS
// vectors and L2 projections.  All arithmetic FP64.
//
// Assembly design.  The reference builds every (3Np)^2 block entry by entry
// at every quadrature point (MAKE_STIFFNESS_VOLUME, assemble_element.f90:24-77;
// MAKE_STIFFNESS_FACE, :404-661).  Here a CTA owns one block and forms, per
// pair of basis functions, plain mass moments over the quadrature points (one
// multiply-add per point), sums them over the tetrahedra or triangles with
// their material and normal factors, and applies the derivatives once per
// block through the Legendre expansion of phi' (k_assemble_self,
// k_assemble_nb): algebraically the reference's sum.

#include "common.cuh"

namespace {

template <int P> struct Deg {
    static constexpr int NP = (P + 1) * (P + 2) * (P + 3) / 6;
    static constexpr int ND = 3 * NP;
    static constexpr int NQ3 = (P + 1) * (P + 1) * (P + 1);
    static constexpr int NQ2 = (P + 1) * (P + 1);
    static constexpr int NPAIR = NP * NP;
};

// Vertex triples of the faces used for normals/areas,
// MAKE_PARTITION_AND_MPI_FILES.f90:1087-1096 (0-based local ids).
__constant__ int c_face_verts[4][3] = {{2, 1, 0}, {0, 1, 3}, {1, 2, 3}, {2, 0, 3}};

// jacobians (Poly_ref_mappings.f90:18-75) and CREATE_NORMAL_FACE
// (MAKE_PARTITION_AND_MPI_FILES.f90:1429-1504), one thread per tetrahedron.
__global__ void k_geometry(int n_tet, const double* __restrict__ X, const int32_t* __restrict__ tv, double* fk,
                           double* jdet, double* nrm, double* area, int* status) {
    int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= n_tet) return;
    double x[4], y[4], z[4];
    for (int v = 0; v < 4; ++v) {
        int id = tv[t * 4 + v];
        x[v] = X[id * 3 + 0]; y[v] = X[id * 3 + 1]; z[v] = X[id * 3 + 2];
    }
    double F[3][4];
    F[0][0] = x[1] - x[0]; F[0][1] = x[2] - x[0]; F[0][2] = x[3] - x[0]; F[0][3] = x[0];
    F[1][0] = y[1] - y[0]; F[1][1] = y[2] - y[0]; F[1][2] = y[3] - y[0]; F[1][3] = y[0];
    F[2][0] = z[1] - z[0]; F[2][1] = z[2] - z[0]; F[2][2] = z[3] - z[0]; F[2][3] = z[0];
    for (int a = 0; a < 3; ++a)
        for (int b = 0; b < 4; ++b) fk[t * 12 + a * 4 + b] = F[a][b];
    double d = F[0][0] * F[1][1] * F[2][2] - F[0][0] * F[1][2] * F[2][1] - F[0][1] * F[1][0] * F[2][2] +
               F[0][1] * F[1][2] * F[2][0] + F[0][2] * F[1][0] * F[2][1] - F[1][1] * F[0][2] * F[2][0];
    jdet[t] = d;
    if (d == 0.0) atomicOr(status, ST_DEGENERATE);
    for (int f = 0; f < 4; ++f) {
        const double* c1 = &X[tv[t * 4 + c_face_verts[f][0]] * 3];
        const double* c2 = &X[tv[t * 4 + c_face_verts[f][1]] * 3];
        const double* c3 = &X[tv[t * 4 + c_face_verts[f][2]] * 3];
        double Qx = c1[0] - c2[0], Qy = c1[1] - c2[1], Qz = c1[2] - c2[2];
        double Px = c3[0] - c2[0], Py = c3[1] - c2[1], Pz = c3[2] - c2[2];
        double n1 = Py * Qz - Pz * Qy, n2 = -Px * Qz + Pz * Qx, n3 = Px * Qy - Py * Qx;
        double nn = sqrt(n1 * n1 + n2 * n2 + n3 * n3);
        if (nn == 0.0) atomicOr(status, ST_DEGENERATE);
        nrm[t * 12 + f * 3 + 0] = n1 / nn;
        nrm[t * 12 + f * 3 + 1] = n2 / nn;
        nrm[t * 12 + f * 3 + 2] = n3 / nn;
        area[t * 4 + f] = nn;
    }
}

// CREATE_BBOX_EL (MAKE_PARTITION_AND_MPI_FILES.f90:1510-1580): bounding box
// and diameter (largest vertex distance) of every polyhedron, a warp each.
// The vertices are gathered once (up to BBOX_V of them, else read again for
// each pair); the root is taken of the largest squared distance, which is the
// largest root since the correctly rounded root is monotone.  A thread per
// polyhedron took 1.17 ms on 11^3 x 6 tets: one dependent chain of loads and
// roots per polyhedron.
constexpr int BBOX_WARPS = 4, BBOX_V = 128;
__global__ void __launch_bounds__(32 * BBOX_WARPS) k_bbox(int n_poly, const int32_t* __restrict__ pptr,
                                                          const int32_t* __restrict__ ptets,
                                                          const int32_t* __restrict__ tv, const double* __restrict__ X,
                                                          double* bbox, double* hk) {
    __shared__ double s_v[BBOX_WARPS][BBOX_V][3];
    const int wid = threadIdx.x >> 5, lane = threadIdx.x & 31, P = blockIdx.x * BBOX_WARPS + wid;
    if (P >= n_poly) return;
    const int t0 = pptr[P], nv = 4 * (pptr[P + 1] - t0);
    const bool fits = nv <= BBOX_V;
    double mn[3] = {1e300, 1e300, 1e300}, mx[3] = {-1e300, -1e300, -1e300};
    for (int a = lane; a < nv; a += 32) {
        const double* c = &X[tv[ptets[t0 + a / 4] * 4 + (a & 3)] * 3];
#pragma unroll
        for (int d = 0; d < 3; ++d) {
            const double v = c[d];
            mn[d] = fmin(mn[d], v);
            mx[d] = fmax(mx[d], v);
            if (fits) s_v[wid][a][d] = v;
        }
    }
    __syncwarp();
    double h2 = 0.0;
    for (int a = lane; a < nv; a += 32) {
        const double* ca = fits ? s_v[wid][a] : &X[tv[ptets[t0 + a / 4] * 4 + (a & 3)] * 3];
        const double a0 = ca[0], a1 = ca[1], a2 = ca[2];
        for (int b = 0; b < a; ++b) {
            const double* cb = fits ? s_v[wid][b] : &X[tv[ptets[t0 + b / 4] * 4 + (b & 3)] * 3];
            h2 = fmax(h2, (a0 - cb[0]) * (a0 - cb[0]) + (a1 - cb[1]) * (a1 - cb[1]) + (a2 - cb[2]) * (a2 - cb[2]));
        }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        h2 = fmax(h2, __shfl_xor_sync(0xffffffffu, h2, o));
#pragma unroll
        for (int d = 0; d < 3; ++d) {
            mn[d] = fmin(mn[d], __shfl_xor_sync(0xffffffffu, mn[d], o));
            mx[d] = fmax(mx[d], __shfl_xor_sync(0xffffffffu, mx[d], o));
        }
    }
    if (lane == 0) {
        for (int d = 0; d < 3; ++d) { bbox[P * 6 + 2 * d] = mn[d]; bbox[P * 6 + 2 * d + 1] = mx[d]; }
        hk[P] = sqrt(h2);
    }
}

// Physical quadrature points of face f of tetrahedron t as basis_boundary
// forms them (basis_function.f90:560-577): temp = Fk node_maps(:,:,f),
// pt = temp nodtria2.
__device__ inline void face_point(const double* fk, const RefTables* ref, int f, int q, double pt[3]) {
    const double* nm = &ref->node_maps[f * 16];
    const double* nt = &ref->nodtria2[q * 4];
    for (int j = 0; j < 3; ++j) {
        double s = 0.0;
        for (int l = 0; l < 4; ++l) {
            double tmp = 0.0;
            for (int m = 0; m < 4; ++m) tmp = tmp + fk[j * 4 + m] * nm[m * 4 + l];
            s = s + tmp * nt[l];
        }
        pt[j] = s;
    }
}

// Shape of the assembly CTAs per degree.  The moments of a self block are
// symmetric, so a CTA owns the NS = Np (Np + 1) / 2 pairs a <= b (packed:
// pair (a, b) at b (b + 1) / 2 + a); a neighbour block owns all Np^2 pairs.
// The thread counts fill whole rounds of pairs with FP64 lanes (the pipe
// retires 2 lanes per clock and SM whether they are used or not): p = 4,
// 630 of 640 and 1225 of 1280 lanes; p = 3, 210 of 224 and 400 of 416.  The face
// integrands are polynomials of degree 2 p, so the triangle rule of the matrix-free
// terms (mf.cu) gives the reference's integrals from 3 / 6 / 12 / 16 points instead
// of 4 / 9 / 16 / 25 (970 polyhedra, p = 4: 3.44 -> 3.03 ms, self blocks 5.24 -> 4.90).
template <int PD> struct AsmShape {
    using D = Deg<PD>;
    static constexpr int NP = D::NP, L1 = PD + 1;
    static constexpr int NS = NP * (NP + 1) / 2;
    static constexpr int T = PD == 4 ? 320 : (PD == 3 ? 224 : (PD == 2 ? 64 : 32));       // self blocks
    static constexpr int PPT = (NS + T - 1) / T;
    static constexpr int R = PD == 4 ? 50 : (PD == 3 ? 64 : (PD == 2 ? 27 : 8));          // tabulated points at once
    static constexpr int FQ = face_rule_points(PD);                                       // points of a face
    static constexpr int FB = R / FQ;                                                     // faces at once
    static constexpr int TN = PD == 4 ? 320 : (PD == 3 ? 416 : (PD == 2 ? 64 : 32));      // neighbour blocks
    static constexpr int PPTN = (D::NPAIR + TN - 1) / TN;
    static_assert(FB >= 1, "one face per table at least");
};

// Position of basis function (x, y, z) in the reference's order, and the
// Legendre expansion of the derivatives: with phi_n the scaled Legendre
// polynomial of degree n on an interval of half width h,
//     phi_n' = (1/h) sum_{m = n-1, n-3, ..} (2m + 1) phi_m,
// at most two terms for n <= 4.  idx[f][k][t] is the basis function of term
// t of d_k phi_f, w[n][t] the weight (2m + 1) (0: no such term).
template <int PD> struct DerTab {
    short idx[Deg<PD>::NP][3][2];
    signed char deg[Deg<PD>::NP][3];
    constexpr DerTab() : idx(), deg() {
        constexpr Blist<PD> BL{};
        int pos[PD + 1][PD + 1][PD + 1] = {};
        for (int f = 0; f < Deg<PD>::NP; ++f) pos[BL.d[f][0]][BL.d[f][1]][BL.d[f][2]] = f;
        for (int f = 0; f < Deg<PD>::NP; ++f)
            for (int k = 0; k < 3; ++k) {
                deg[f][k] = (signed char)BL.d[f][k];
                for (int t = 0; t < 2; ++t) {
                    int q[3] = {BL.d[f][0], BL.d[f][1], BL.d[f][2]};
                    q[k] -= 1 + 2 * t;
                    idx[f][k][t] = (short)(q[k] >= 0 ? pos[q[0]][q[1]][q[2]] : 0);
                }
            }
    }
};
template <int PD> __device__ const DerTab<PD> g_der{};
// Its copy in shared memory (the threads of a warp read different functions).
template <int PD> __device__ __forceinline__ void load_der(DerTab<PD>* dst) {
    static_assert(sizeof(DerTab<PD>) % sizeof(short) == 0, "copied as shorts");
    const short* src = reinterpret_cast<const short*>(&g_der<PD>);
    for (int i = threadIdx.x; i < (int)(sizeof(DerTab<PD>) / sizeof(short)); i += blockDim.x)
        reinterpret_cast<short*>(dst)[i] = src[i];
}
// The weights of a box: w[f][k][t] = scale (2m + 1) / h_k for term t of d_k phi_f,
// m = n_k - 1 - 2t (0: no such term), formed once per CTA: a division per term
// and pair cost more than the expansion itself.
template <int PD> __device__ __forceinline__ void load_weights(const DerTab<PD>& der, const double* hb, double scale, double* w) {
    for (int i = threadIdx.x; i < Deg<PD>::NP * 6; i += blockDim.x) {
        const int f = i / 6, k = i % 6 / 2, m = der.deg[f][k] - 1 - 2 * (i % 2);
        w[i] = m >= 0 ? scale * (double)(2 * m + 1) / hb[k] : 0.0;
    }
}

struct AsmArgs {
    const int32_t* row_ptr;
    const int32_t* blk_row;
    const int32_t* col;
    const int64_t* bf_ptr;
    const int32_t* bf;
    const int32_t* poly_ptr;
    const int32_t* poly_tets;
    const int32_t* tet_poly;
    const int32_t* tet_mat;
    const int32_t* neigh;
    const double* mat;
    const double* fk;
    const double* jdet;
    const double* nrm;
    const double* area;
    const double* bbox;
    const double* hk;
    const RefTables* ref;
    double alpha, theta;
    double* out;      // [n_blocks][ND][ND], each block column-major
    double* M;        // [n_poly][NP][NP] rho-weighted mass (may be null)
    double* Mm;       // unweighted (modal) mass
    int64_t block0;   // first block of this launch (neighbour blocks)
};

// Interval constants of a bounding box per coordinate, as legendre_1d forms them.
struct BoxC {
    double mb[3], hb[3], ih[3], is[3];   // ih: 1 / hb, is: 1 / sqrt(hb)
    double il[3], sl[3];                 // what ih and is lack of the exact reciprocals
};
__device__ __forceinline__ void box_consts(const double* bb, BoxC* B, int d) {
    B->hb[d] = (bb[2 * d + 1] - bb[2 * d]) / 2.0;
    B->mb[d] = (bb[2 * d + 1] + bb[2 * d]) / 2.0;
    const double sh = sqrt(B->hb[d]);
    B->ih[d] = 1.0 / B->hb[d];
    B->is[d] = 1.0 / sh;
    B->il[d] = fma(-B->hb[d], B->ih[d], 1.0) * B->ih[d];
    B->sl[d] = fma(-sh, B->is[d], 1.0) * B->is[d];
}
// a / b for a known b: zh = 1 / b rounded, zl the rest.  The sum before its one
// rounding is off by 2^-105 of the quotient, so the result is the division's but
// for quotients closer than that to a midpoint (Brisebarre, Muller and Raina,
// "Accelerating correctly rounded floating-point division when the divisor is
// known in advance", IEEE Trans. Computers 53(8), 2004): two FP64 operations
// instead of a division's nine or so.
__device__ __forceinline__ double div_known(double a, double zh, double zl) { return fma(a, zh, a * zl); }
// The scaled Legendre values of degrees 0..PD at coordinate x of direction d:
// legendre_1d's values, with the interval's constants and the normalised
// coordinate formed once for all degrees, and its divisions by them in two
// operations each (projection of 10,123
// polyhedra at p = 4: 14.5 -> 12.4 ms).
template <int PD>
__device__ __forceinline__ void legendre_vals(const BoxC* B, int d, double x, double* v) {
    const double xp = div_known(x - B->mb[d], B->ih[d], B->il[d]), sh = B->is[d], sl = B->sl[d];
    v[0] = sh;
#pragma unroll
    for (int n = 1; n <= PD; ++n) v[n] = div_known(lp_nonnorm(xp, n), sh, sl);
}

// The same to rounding, for the operator blocks: the three-term recurrence and
// products with the interval's reciprocals instead of a division per degree
// (ih = 1 / hb, is = 1 / sqrt(hb)).
template <int PD>
__device__ __forceinline__ void legendre_rec(double mb, double ih, double is, double x, double* v) {
    const double xp = (x - mb) * ih;
    double l0 = is, l1 = xp * is;
    v[0] = l0;
    v[1] = l1;
#pragma unroll
    for (int n = 1; n < PD; ++n) {
        const double l2 = fma((2.0 * n + 1.0) / (n + 1.0) * xp, l1, -(n / (n + 1.0)) * l0);
        v[n + 1] = l2;
        l0 = l1;
        l1 = l2;
    }
}

// Coordinate j of the affine map of face f of a tetrahedron: cm[l] =
// (Fk node_maps(:,:,f))(j, l), as face_point forms it.
__device__ __forceinline__ double face_map(const double* fk, const RefTables* ref, int f, int j, int l) {
    const double* nm = &ref->node_maps[f * 16];
    double tmp = 0.0;
    for (int m = 0; m < 4; ++m) tmp = tmp + fk[j * 4 + m] * nm[m * 4 + l];
    return tmp;
}

// The 12 factors of a face's moments P(a, b) = sum_q W phi_a phi_b, W =
// weight * area: c lambda n_j, c mu n_j (j = 0..2) and sigma T_ij for (i, j)
// = 00, 11, 22, 01, 02, 12 (T_ii = n_i^2 + (n_j^2 + n_k^2) / 2, T_ij =
// n_i n_j / 2).
constexpr int FACE_F = 12;
__device__ __forceinline__ void face_factors(const AsmArgs& A, int code, int P, int Qn, double c, double pdeg2, double* o) {
    const int t = code >> 2, f = code & 3;
    const int mid = A.tet_mat[t];
    const double lam = A.mat[mid * 3 + 1], mu = A.mat[mid * 3 + 2];
    const double* n = &A.nrm[t * 12 + f * 3];
    const double h1 = A.hk[P];
    const double sigma = A.alpha * pdeg2 / (Qn < 0 ? h1 : fmin(h1, A.hk[Qn])) * (lam + 2 * mu);
    const double n2[3] = {n[0] * n[0], n[1] * n[1], n[2] * n[2]};
#pragma unroll
    for (int j = 0; j < 3; ++j) {
        o[j] = c * lam * n[j];
        o[3 + j] = c * mu * n[j];
        o[6 + j] = sigma * (n2[j] + 0.5 * n2[(j + 1) % 3] + 0.5 * n2[(j + 2) % 3]);
    }
    o[9] = sigma * (0.5 * n[0] * n[1]);
    o[10] = sigma * (0.5 * n[0] * n[2]);
    o[11] = sigma * (0.5 * n[1] * n[2]);
}

enum { ASM_MASS = 0, ASM_K = 1, ASM_ADG = 2 };

// The self block of each polyhedron (stiffness or DG-norm block) and its two
// mass matrices, one CTA per polyhedron.
//
// FP64-pipe bound, so the design removes FP64 operations.  Derivatives of
// Legendre products are sums of at most two lower ones per direction, so
// every term follows from plain mass moments: per tetrahedron M_t(a, b) =
// sum_q w phi_a phi_b (needed for the mass matrices anyway), per face
// P(a, b) = sum_q W phi_a phi_b, each weighted with its material and normal
// factors and summed over the tetrahedra or faces; only then the derivative
// expansion is applied, once per block:
//     volume  V_ij = D_i (sum lambda M_t) D_j^T + D_j (sum mu M_t) D_i^T + delta_ij sum_k D_k (sum mu M_t) D_k^T
//     faces   S = sum sigma T_ij P,  H-terms D_i (sum c lambda n_j P), ...
// A quadrature point of a pair then costs one multiply-add instead of ten
// (volume) or seven (faces).  All moments are symmetric, so only a <= b is
// formed.  The mass matrices keep legendre_1d's values and the sums' order
// (products and sums rounded separately), because their inverses amplify a
// change of rounding by the condition number (up to 1e7).
template <int PD, int WHICH>
__global__ void __launch_bounds__(AsmShape<PD>::T) k_assemble_self(AsmArgs A) {
    using D = Deg<PD>;
    using S = AsmShape<PD>;
    constexpr int NP = D::NP, ND = D::ND, NQ3 = D::NQ3, NQ2 = S::FQ, NS = S::NS, T = S::T, PPT = S::PPT, R = S::R,
                  L1 = S::L1, FB = S::FB;
    constexpr int NMAT = WHICH == ASM_MASS ? 0 : 14;   // lambda M, mu M, c lambda n_j P (3), c mu n_j P (3), sigma T P (6)
    extern __shared__ double sm[];
    double* mats = sm;                    // [NMAT][NS]
    double* tphi = mats + NMAT * NS;      // [R][NP]
    double* twphi = tphi + R * NP;        // [R][NP]
    double* tleg = twphi + R * NP;        // [R][3][L1]
    double* tw = tleg + R * 3 * L1;       // [R]
    double* ffac = tw + R;                // [FB][FACE_F]
    double* fmap = ffac + FB * FACE_F;    // [FB][3][4]
    __shared__ BoxC box;
    __shared__ DerTab<PD> der;
    const int tid = threadIdx.x, P = blockIdx.x;
    load_der<PD>(&der);
    if (tid < 3) box_consts(&A.bbox[P * 6], &box, tid);
    int pm[PPT], pn[PPT];                 // this thread's pairs m <= n
#pragma unroll
    for (int u = 0; u < PPT; ++u) {
        const int e = tid + u * T;
        int n = 0;
        while ((n + 1) * (n + 2) / 2 <= e) ++n;
        pn[u] = n < NP ? n : NP - 1;
        pm[u] = n < NP ? e - n * (n + 1) / 2 : 0;
    }
    // products of the 1-D factors at r0 points, in basis_eval's order
    auto products = [&](int r0) {
        for (int it = tid; it < r0 * NP; it += T) {
            const int q = it / NP, f = it - q * NP;
            const double* tq = tleg + q * 3 * L1;
            const double ph = tq[der.deg[f][0]] * tq[L1 + der.deg[f][1]] * tq[2 * L1 + der.deg[f][2]];
            tphi[it] = ph;
            twphi[it] = tw[q] * ph;
        }
    };
    // ---- mass moments of the sub-tetrahedra ----
    double msum[PPT], mrho[PPT], mlam[PPT], mmu[PPT];
#pragma unroll
    for (int u = 0; u < PPT; ++u) msum[u] = mrho[u] = mlam[u] = mmu[u] = 0.0;
    for (int kt = A.poly_ptr[P]; kt < A.poly_ptr[P + 1]; ++kt) {
        const int t = A.poly_tets[kt];
        const double* fk = &A.fk[t * 12];
        const int mid = A.tet_mat[t];
        const double rho = A.mat[mid * 3 + 0], lam = A.mat[mid * 3 + 1], mu = A.mat[mid * 3 + 2];
        const double aj = fabs(A.jdet[t]);
        double Mt[PPT];
#pragma unroll
        for (int u = 0; u < PPT; ++u) Mt[u] = 0.0;
        for (int q0 = 0; q0 < NQ3; q0 += R) {
            const int nq = (NQ3 - q0) < R ? (NQ3 - q0) : R;
            __syncthreads();
            for (int it = tid; it < nq * 3; it += T) {
                const int qq = it / 3, d = it - qq * 3;
                const double* nt = &A.ref->nodtet3[(q0 + qq) * 4];
                double x = 0.0;
                for (int l = 0; l < 4; ++l) x = x + fk[d * 4 + l] * nt[l];
                legendre_vals<PD>(&box, d, x, tleg + it * L1);
                if (d == 0) tw[qq] = A.ref->weitet3[q0 + qq] * aj;
            }
            __syncthreads();
            products(nq);
            __syncthreads();
            for (int qq = 0; qq < nq; ++qq)
#pragma unroll
                for (int u = 0; u < PPT; ++u) Mt[u] += twphi[qq * NP + pm[u]] * tphi[qq * NP + pn[u]];
        }
#pragma unroll
        for (int u = 0; u < PPT; ++u) {
            msum[u] += Mt[u];
            mrho[u] += Mt[u] * rho;
            if (WHICH != ASM_MASS) {
                mlam[u] = fma(Mt[u], lam, mlam[u]);
                mmu[u] = fma(Mt[u], mu, mmu[u]);
            }
        }
    }
#pragma unroll
    for (int u = 0; u < PPT; ++u) {
        const int e = tid + u * T;
        if (e < NS) {
            if (A.M != nullptr) {
                double* M = A.M + (int64_t)P * D::NPAIR;
                double* Mm = A.Mm + (int64_t)P * D::NPAIR;
                M[pm[u] * NP + pn[u]] = M[pn[u] * NP + pm[u]] = mrho[u];
                Mm[pm[u] * NP + pn[u]] = Mm[pn[u] * NP + pm[u]] = msum[u];
            }
            if (WHICH != ASM_MASS) {
                mats[e] = mlam[u];
                mats[NS + e] = mmu[u];
            }
        }
    }
    if constexpr (WHICH != ASM_MASS) {
        // ---- face moments ----
        const int64_t k = A.row_ptr[P];   // the self block comes first in its row
        double acc[PPT][FACE_F];
#pragma unroll
        for (int u = 0; u < PPT; ++u)
#pragma unroll
            for (int j = 0; j < FACE_F; ++j) acc[u][j] = 0.0;
        const int64_t e0 = A.bf_ptr[k], e1 = A.bf_ptr[k + 1];
        for (int64_t eb = e0; eb < e1; eb += FB) {
            const int nf = (int)((e1 - eb) < FB ? (e1 - eb) : FB);
            __syncthreads();
            for (int it = tid; it < nf * 12; it += T) {
                const int fi = it / 12, jl = it - fi * 12, code = A.bf[eb + fi];
                fmap[it] = face_map(&A.fk[(code >> 2) * 12], A.ref, code & 3, jl / 4, jl & 3);
            }
            for (int fi = tid; fi < nf; fi += T) {
                const int code = A.bf[eb + fi], e2 = A.neigh[code];
                const bool dir = e2 == LYMPH_BC_DIRI;
                face_factors(A, code, P, dir ? -1 : A.tet_poly[e2], dir ? 1.0 : 0.5, (double)(PD * PD), ffac + fi * FACE_F);
            }
            __syncthreads();
            for (int it = tid; it < nf * NQ2 * 3; it += T) {
                const int qq = it / 3, d = it - qq * 3, fi = qq / NQ2, q = qq - fi * NQ2;
                const double* cm = fmap + fi * 12 + d * 4;
                const double* nt = &A.ref->facenod[q * 4];
                double x = 0.0;
                for (int l = 0; l < 4; ++l) x = x + cm[l] * nt[l];
                legendre_rec<PD>(box.mb[d], box.ih[d], box.is[d], x, tleg + it * L1);
                if (d == 0) tw[qq] = A.ref->facewei[q] * A.area[A.bf[eb + fi]];
            }
            __syncthreads();
            products(nf * NQ2);
            __syncthreads();
            for (int fi = 0; fi < nf; ++fi) {
                double p[PPT];
#pragma unroll
                for (int u = 0; u < PPT; ++u) p[u] = 0.0;
                for (int q = fi * NQ2; q < (fi + 1) * NQ2; ++q)
#pragma unroll
                    for (int u = 0; u < PPT; ++u) p[u] = fma(twphi[q * NP + pm[u]], tphi[q * NP + pn[u]], p[u]);
#pragma unroll
                for (int u = 0; u < PPT; ++u)
#pragma unroll
                    for (int j = (WHICH == ASM_ADG ? 6 : 0); j < FACE_F; ++j)
                        acc[u][j] = fma(ffac[fi * FACE_F + j], p[u], acc[u][j]);
            }
        }
#pragma unroll
        for (int u = 0; u < PPT; ++u) {
            const int e = tid + u * T;
            if (e < NS)
#pragma unroll
                for (int j = (WHICH == ASM_ADG ? 6 : 0); j < FACE_F; ++j) mats[(2 + j) * NS + e] = acc[u][j];
        }
        __syncthreads();                     // the last faces' tables are read
        double* wder = tphi;                 // [NP][3][2], over them
        load_weights<PD>(der, box.hb, 1.0, wder);
        __syncthreads();
        // ---- the block from the moments, written column-major ----
        const double* ML = mats;
        const double* MM = mats + NS;
        const double* PL = mats + 2 * NS;    // [3][NS]
        const double* PM = mats + 5 * NS;    // [3][NS]
        const double* SP = mats + 8 * NS;    // [6][NS]
        auto sym = [](int a, int b) { return a <= b ? b * (b + 1) / 2 + a : a * (a + 1) / 2 + b; };
        double* o = A.out + k * ND * ND;
        for (int pr = tid; pr < D::NPAIR; pr += T) {
            const int b = pr / NP, a = pr - b * NP;
            int ia[3][2], ib[3][2];
            double wa[3][2], wb[3][2];
#pragma unroll
            for (int d = 0; d < 3; ++d)
#pragma unroll
                for (int t = 0; t < 2; ++t) {
                    ia[d][t] = der.idx[a][d][t];
                    ib[d][t] = der.idx[b][d][t];
                    wa[d][t] = wder[a * 6 + d * 2 + t];
                    wb[d][t] = wder[b * 6 + d * 2 + t];
                }
            double V[3][3], tr = 0.0;        // lambda D_i M D_j^T + mu D_j M D_i^T
            double Gm[3][3];
#pragma unroll
            for (int i = 0; i < 3; ++i)
#pragma unroll
                for (int j = 0; j < 3; ++j) {
                    double gl = 0.0, gm = 0.0;
#pragma unroll
                    for (int t = 0; t < 2; ++t)
#pragma unroll
                        for (int s = 0; s < 2; ++s) {
                            const double w = wa[i][t] * wb[j][s];
                            if (w != 0.0) {
                                const int x = sym(ia[i][t], ib[j][s]);
                                gl = fma(w, ML[x], gl);
                                gm = fma(w, MM[x], gm);
                            }
                        }
                    V[i][j] = gl;
                    Gm[i][j] = gm;
                }
            tr = Gm[0][0] + Gm[1][1] + Gm[2][2];
#pragma unroll
            for (int i = 0; i < 3; ++i)
#pragma unroll
                for (int j = 0; j < 3; ++j) V[i][j] += Gm[j][i] + (i == j ? tr : 0.0);
            const int e = sym(a, b);
            const double s01 = SP[3 * NS + e], s02 = SP[4 * NS + e], s12 = SP[5 * NS + e];
            V[0][0] += SP[e]; V[1][1] += SP[NS + e]; V[2][2] += SP[2 * NS + e];
            V[0][1] += s01; V[1][0] += s01;
            V[0][2] += s02; V[2][0] += s02;
            V[1][2] += s12; V[2][1] += s12;
            if (WHICH == ASM_K) {
                // theta I(i,j,a,b) - I(j,i,b,a), I(i,j) = D_i PL_j + D_j PM_i + delta_ij sum_k D_k PM_k
                double tL = 0.0, tR = 0.0;
                double L[3][3], Rr[3][3];
#pragma unroll
                for (int i = 0; i < 3; ++i)
#pragma unroll
                    for (int j = 0; j < 3; ++j) L[i][j] = Rr[i][j] = 0.0;
#pragma unroll
                for (int i = 0; i < 3; ++i)
#pragma unroll
                    for (int t = 0; t < 2; ++t) {
                        if (wa[i][t] != 0.0) {
                            const int x = sym(ia[i][t], b);
#pragma unroll
                            for (int j = 0; j < 3; ++j) {
                                L[i][j] = fma(wa[i][t], PL[j * NS + x], L[i][j]);
                                L[j][i] = fma(wa[i][t], PM[j * NS + x], L[j][i]);
                            }
                            tL = fma(wa[i][t], PM[i * NS + x], tL);
                        }
                        if (wb[i][t] != 0.0) {
                            const int x = sym(a, ib[i][t]);
#pragma unroll
                            for (int j = 0; j < 3; ++j) {
                                Rr[j][i] = fma(wb[i][t], PL[j * NS + x], Rr[j][i]);
                                Rr[i][j] = fma(wb[i][t], PM[j * NS + x], Rr[i][j]);
                            }
                            tR = fma(wb[i][t], PM[i * NS + x], tR);
                        }
                    }
#pragma unroll
                for (int i = 0; i < 3; ++i)
#pragma unroll
                    for (int j = 0; j < 3; ++j) {
                        double l = L[i][j], r = Rr[i][j];
                        if (i == j) { l += tL; r += tR; }
                        V[i][j] += A.theta * l - r;
                    }
            }
#pragma unroll
            for (int i = 0; i < 3; ++i)
#pragma unroll
                for (int j = 0; j < 3; ++j) o[(int64_t)(j * NP + b) * ND + i * NP + a] = V[i][j];
        }
    }
}

// One neighbour block K_PQ = -theta/2 I - S - IT/2 per CTA (or the DG norm's
// -S), from the moments P(a, b) = sum_q W phi^P_a phi^Q_b of the triangles P
// shares with Q, as in k_assemble_self: 16 multiply-adds per triangle and
// pair for the moment (p = 4; 25 with the reference's rule), 12 for its weighted sums, and the derivative
// expansion once per block,
//     I(i,j)  = D_i PL_j + D_j PM_i + delta_ij sum_k D_k PM_k,
//     IT(i,j) = PL_j D_i^T + PM_i D_j^T + delta_ij sum_k PM_k D_k^T
// (IT carries the reference's index order, assemble_element.f90:610-616),
// PL_j = sum lambda n_j P, PM_j = sum mu n_j P, D on the left in P's basis and
// on the right in Q's.
template <int PD, int WHICH>
__global__ void __launch_bounds__(AsmShape<PD>::TN, PD == 4 ? 2 : 1) k_assemble_nb(AsmArgs A) {
    using D = Deg<PD>;
    using S = AsmShape<PD>;
    constexpr int NP = D::NP, ND = D::ND, NQ2 = S::FQ, NPAIR = D::NPAIR, T = S::TN, PPT = S::PPTN, L1 = S::L1;
    extern __shared__ double sm[];
    double* PL = sm;                                     // [3][NPAIR], pair (a, b) at b NP + a
    double* PM = PL + (WHICH == ASM_K ? 3 * NPAIR : 0);  // [3][NPAIR]
    double* fphi = PM + (WHICH == ASM_K ? 3 * NPAIR : 0);   // [2][NQ2][NP]; Q's side carries W
    double* tleg = fphi + 2 * NQ2 * NP;                  // [2][NQ2][3][L1]
    double* ffac = tleg + 2 * NQ2 * 3 * L1;              // [FACE_F]
    double* fmap = ffac + FACE_F;                        // [3][4]
    __shared__ BoxC box[2];
    const int tid = threadIdx.x;
    const int64_t k = A.block0 + blockIdx.x;
    const int P = A.blk_row[k], Q = A.col[k];
    if (P == Q) return;                                  // self blocks: k_assemble_self
    __shared__ DerTab<PD> der;
    load_der<PD>(&der);
    if (tid < 6) box_consts(&A.bbox[(tid < 3 ? P : Q) * 6], &box[tid / 3], tid % 3);
    double SP[PPT][6];
#pragma unroll
    for (int u = 0; u < PPT; ++u)
#pragma unroll
        for (int j = 0; j < 6; ++j) SP[u][j] = 0.0;
    const int64_t e0 = A.bf_ptr[k], e1 = A.bf_ptr[k + 1];
    for (int64_t e = e0; e < e1; ++e) {
        const int code = A.bf[e];
        __syncthreads();
        if (tid < 12) fmap[tid] = face_map(&A.fk[(code >> 2) * 12], A.ref, code & 3, tid / 4, tid & 3);
        if (tid == T - 1) face_factors(A, code, P, Q, 1.0, (double)(PD * PD), ffac);
        __syncthreads();
        for (int it = tid; it < 2 * NQ2 * 3; it += T) {
            const int s = it / (NQ2 * 3), r = it - s * NQ2 * 3, q = r / 3, d = r - q * 3;
            const double* cm = fmap + d * 4;
            const double* nt = &A.ref->facenod[q * 4];
            double x = 0.0;
            for (int l = 0; l < 4; ++l) x = x + cm[l] * nt[l];
            legendre_rec<PD>(box[s].mb[d], box[s].ih[d], box[s].is[d], x, tleg + it * L1);
        }
        __syncthreads();
        const double ar = A.area[code];
        for (int it = tid; it < 2 * NQ2 * NP; it += T) {
            const int s = it / (NQ2 * NP), r = it - s * NQ2 * NP, q = r / NP, f = r - q * NP;
            const double* tq = tleg + (s * NQ2 + q) * 3 * L1;
            double ph = tq[der.deg[f][0]] * tq[L1 + der.deg[f][1]] * tq[2 * L1 + der.deg[f][2]];
            if (s == 1) ph *= A.ref->facewei[q] * ar;
            fphi[it] = ph;
        }
        __syncthreads();
        double p[PPT];
#pragma unroll
        for (int u = 0; u < PPT; ++u) p[u] = 0.0;
        int ra[PPT], rb[PPT];
#pragma unroll
        for (int u = 0; u < PPT; ++u) {
            const int pr = tid + u * T < NPAIR ? tid + u * T : NPAIR - 1;
            rb[u] = pr / NP;
            ra[u] = pr - rb[u] * NP;
        }
        for (int q = 0; q < NQ2; ++q)
#pragma unroll
            for (int u = 0; u < PPT; ++u) p[u] = fma(fphi[q * NP + ra[u]], fphi[(NQ2 + q) * NP + rb[u]], p[u]);
#pragma unroll
        for (int u = 0; u < PPT; ++u) {
            const int pr = tid + u * T;
            if (pr >= NPAIR) continue;
            if (WHICH == ASM_K) {
#pragma unroll
                for (int j = 0; j < 3; ++j) {
                    // each thread owns its pairs, so the sums over the triangles need no barrier
                    PL[j * NPAIR + pr] = e == e0 ? ffac[j] * p[u] : fma(ffac[j], p[u], PL[j * NPAIR + pr]);
                    PM[j * NPAIR + pr] = e == e0 ? ffac[3 + j] * p[u] : fma(ffac[3 + j], p[u], PM[j * NPAIR + pr]);
                }
            }
#pragma unroll
            for (int j = 0; j < 6; ++j) SP[u][j] = fma(ffac[6 + j], p[u], SP[u][j]);
        }
    }
    double* wder = fphi;                                 // [2][NP][3][2], over the tables
    static_assert(2 * NP * 6 <= 2 * NQ2 * NP + 2 * NQ2 * 3 * L1, "the weights fit the tables");
    __syncthreads();   // the last triangle's tables are read
    if (WHICH == ASM_K) {
        load_weights<PD>(der, box[0].hb, -0.5 * A.theta, wder);
        load_weights<PD>(der, box[1].hb, -0.5, wder + NP * 6);
    }
    __syncthreads();
    double* o = A.out + k * ND * ND;
#pragma unroll
    for (int u = 0; u < PPT; ++u) {
        const int pr = tid + u * T;
        if (pr >= NPAIR) continue;
        const int b = pr / NP, a = pr - b * NP;
        double V[3][3];
        V[0][0] = -SP[u][0]; V[1][1] = -SP[u][1]; V[2][2] = -SP[u][2];
        V[0][1] = V[1][0] = -SP[u][3];
        V[0][2] = V[2][0] = -SP[u][4];
        V[1][2] = V[2][1] = -SP[u][5];
        if (WHICH == ASM_K) {
            double tr = 0.0;
#pragma unroll
            for (int i = 0; i < 3; ++i)
#pragma unroll
                for (int t = 0; t < 2; ++t) {
                    const double wl = wder[a * 6 + i * 2 + t];
                    if (wl != 0.0) {
                        const int x = b * NP + der.idx[a][i][t];
#pragma unroll
                        for (int j = 0; j < 3; ++j) {
                            V[i][j] = fma(wl, PL[j * NPAIR + x], V[i][j]);
                            V[j][i] = fma(wl, PM[j * NPAIR + x], V[j][i]);
                        }
                        tr = fma(wl, PM[i * NPAIR + x], tr);
                    }
                    const double wr = wder[(NP + b) * 6 + i * 2 + t];
                    if (wr != 0.0) {
                        const int x = der.idx[b][i][t] * NP + a;
#pragma unroll
                        for (int j = 0; j < 3; ++j) {
                            V[i][j] = fma(wr, PL[j * NPAIR + x], V[i][j]);
                            V[j][i] = fma(wr, PM[j * NPAIR + x], V[j][i]);
                        }
                        tr = fma(wr, PM[i * NPAIR + x], tr);
                    }
                }
            V[0][0] += tr; V[1][1] += tr; V[2][2] += tr;
        }
#pragma unroll
        for (int i = 0; i < 3; ++i)
#pragma unroll
            for (int j = 0; j < 3; ++j) o[(int64_t)(j * NP + b) * ND + i * NP + a] = V[i][j];
    }
}

template <int PD, int WHICH> size_t asm_self_smem() {
    using S = AsmShape<PD>;
    constexpr int nmat = WHICH == ASM_MASS ? 0 : 14;
    return sizeof(double) * ((size_t)nmat * S::NS + 2 * (size_t)S::R * S::NP + (size_t)S::R * 3 * S::L1 + S::R +
                             S::FB * (FACE_F + 12));
}
template <int PD, int WHICH> size_t asm_nb_smem() {
    using S = AsmShape<PD>;
    constexpr int NQ2 = S::FQ;
    return sizeof(double) * ((WHICH == ASM_K ? 6 * (size_t)Deg<PD>::NPAIR : 0) + 2 * (size_t)NQ2 * S::NP +
                             2 * (size_t)NQ2 * 3 * S::L1 + FACE_F + 12);
}

// cholesky (vet_mat_operations.f90:84-120) of the NP x NP matrix of every
// polyhedron, one warp each; writes R (row-major upper).
__global__ void k_cholesky(int n_poly, int NP, const double* __restrict__ A, double* R, int* status) {
    const int warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
    if (warp >= n_poly) return;
    extern __shared__ double shm[];
    double* r = shm + (threadIdx.x >> 5) * NP * NP;
    const double* a = A + (int64_t)warp * NP * NP;
    for (int i = lane; i < NP * NP; i += 32) r[i] = 0.0;
    __syncwarp();
    bool ok = true;
    for (int j = 0; j < NP; ++j) {
        // row j's sums, the diagonal's (lane 0 of the first round) beside the
        // others: alone, it doubled the chain of FP64 operations
        double rjj = 1.0;
        for (int i0 = j; i0 < NP; i0 += 32) {
            const int i = i0 + lane;
            double s = i < NP ? a[j * NP + i] : 1.0;
            if (i < NP)
                for (int kk = 0; kk < j; ++kk) s = s - r[kk * NP + j] * r[kk * NP + i];
            if (i0 == j) {
                double sum = __shfl_sync(0xffffffffu, s, 0);
                if (!(sum > 0.0)) { ok = false; sum = 1.0; }
                rjj = sqrt(sum);
            }
            if (i < NP) r[j * NP + i] = i == j ? rjj : s / rjj;
        }
        __syncwarp();
    }
    if (!ok && lane == 0) atomicOr(status, ST_NOT_SPD);
    for (int i = lane; i < NP * NP; i += 32) R[(int64_t)warp * NP * NP + i] = r[i];
}

// Inverse from a Cholesky factor: column k of the inverse is solve_LU(R^T, R,
// e_k) (vet_mat_operations.f90:123-153, reference operation order), one lane
// per column.  Stored column-major: inv[c*NP + r], so that lane r of a warp
// reads consecutive addresses when applying it.  INV_MATS factors per CTA
// come into shared memory with the columns being solved (NP <= MAX_NP); a
// fifth warp solves the columns beyond 31 of all of them, which otherwise
// cost each matrix a second pass of the whole chain for three lanes.
constexpr int INV_MATS = 4, INV_THREADS = 32 * (INV_MATS + 1);
__global__ void __launch_bounds__(INV_THREADS) k_mass_inverse(int n_poly, int NP, const double* __restrict__ R, double* Minv) {
    extern __shared__ double shm[];
    const int NP2 = NP * NP, tid = threadIdx.x, P0 = blockIdx.x * INV_MATS;
    const int nm = n_poly - P0 < INV_MATS ? n_poly - P0 : INV_MATS;
    double *s_r = shm, *s_x = shm + INV_MATS * NP2;   // factors; columns as [row][column]
    for (int i = tid; i < nm * NP2; i += INV_THREADS) s_r[i] = R[(int64_t)P0 * NP2 + i];
    __syncthreads();
    const int wid = tid >> 5, lane = tid & 31, rest = NP > 32 ? NP - 32 : 0;
    const int mat = wid < INV_MATS ? wid : (rest ? lane / rest : INV_MATS);
    const int k = wid < INV_MATS ? lane : (rest ? 32 + lane % rest : NP);
    if (mat < nm && k < NP) {
        const double* r = s_r + mat * NP2;
        double* x = s_x + mat * NP2 + k;
        for (int i = 0; i < NP; ++i) {
            double y = (i == k) ? 1.0 : 0.0;
            for (int j = 0; j < i; ++j) y = y - r[j * NP + i] * x[j * NP];
            x[i * NP] = y / r[i * NP + i];
        }
        for (int i = NP - 1; i >= 0; --i) {
            double v = x[i * NP];
            for (int j = i + 1; j < NP; ++j) v = v - r[i * NP + j] * x[j * NP];
            x[i * NP] = v / r[i * NP + i];
        }
    }
    __syncthreads();
    for (int i = tid; i < nm * NP2; i += INV_THREADS) {
        const int m = i / NP2, e = i - m * NP2, c = e / NP, row = e - c * NP;
        Minv[(int64_t)P0 * NP2 + i] = s_x[m * NP2 + row * NP + c];
    }
}

// The same for the larger factors of the absorbing polyhedra (size 3 Np): the
// columns are solved in place in device memory.
__global__ void k_inverse_columns(int n, int NP, const double* __restrict__ R, double* inv) {
    const int warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
    if (warp >= n) return;
    const double* r = R + (int64_t)warp * NP * NP;
    double* out = inv + (int64_t)warp * NP * NP;
    for (int k = lane; k < NP; k += 32) {
        double* x = out + (int64_t)k * NP;  // column k, solved in place
        for (int i = 0; i < NP; ++i) x[i] = (i == k) ? 1.0 : 0.0;
        for (int i = 0; i < NP; ++i) {
            double y = x[i];
            for (int j = 0; j < i; ++j) y = y - r[j * NP + i] * x[j];
            x[i] = y / r[i * NP + i];
        }
        for (int i = NP - 1; i >= 0; --i) {
            double v = x[i];
            for (int j = i + 1; j < NP; ++j) v = v - r[i * NP + j] * x[j];
            x[i] = v / r[i * NP + i];
        }
    }
}

// ---- data functions (problem_data_and_properties.f90) ----
// Each takes sn[d] = sin(pi x_d), cs[d] = cos(pi x_d) of the point, formed
// once per point and coordinate; the products keep the reference's order.
constexpr double DATA_PI = 3.141592653589793;

__device__ inline void dev_u_space(const double* sn, const double* cs, double r[3]) {
    r[0] = cs[0] * sn[1] * sn[2];
    r[1] = sn[0] * cs[1] * sn[2];
    r[2] = sn[0] * sn[1] * cs[2];
}

__device__ inline void dev_forcing(int id, double lam, double mu, double rho, const double* sn, const double* cs,
                                   double r[3]) {
    const double PI = DATA_PI;
    if (id == LYMPH_F_TIME) {
        const double c = (-2.0 * rho + 3.0 * (lam + 2.0 * mu)) * PI * PI;
        r[0] = c * cs[0] * sn[1] * sn[2];
        r[1] = c * sn[0] * cs[1] * sn[2];
        r[2] = c * sn[0] * sn[1] * cs[2];
    } else if (id == LYMPH_F_STAT) {
        r[0] = 3 * PI * PI * cs[0] * sn[1] * sn[2] * (lam + 2 * mu);
        r[1] = 3 * PI * PI * cs[1] * sn[0] * sn[2] * (lam + 2 * mu);
        r[2] = 3 * PI * PI * cs[2] * sn[0] * sn[1] * (lam + 2 * mu);
    } else {
        r[0] = r[1] = r[2] = 0.0;
    }
}

__device__ inline void dev_dirichlet(int id, int tag, const double* sn, const double* cs, double r[3]) {
    if (id == LYMPH_GD) {
        if (tag == 1 || tag == 2 || tag == 3) dev_u_space(sn, cs, r);
        else r[0] = r[1] = r[2] = 0.0;
    } else if (id == LYMPH_GD_STAT) {
        r[0] = r[1] = r[2] = 2.0;
    } else {
        r[0] = r[1] = r[2] = 0.0;
    }
}

__device__ inline void dev_neumann(int id, double lam, double mu, const double n[3], int tag, const double* sn,
                                   const double* cs, double r[3]) {
    const double PI = DATA_PI;
    r[0] = r[1] = r[2] = 0.0;
    if (id != LYMPH_GN || !(tag == 1 || tag == 2 || tag == 3)) return;
    double s[3][3];
    const double d = -PI * sn[0] * sn[1] * sn[2] * (3.0 * lam + 2.0 * mu);
    s[0][0] = d; s[1][1] = d; s[2][2] = d;
    s[0][1] = 2.0 * mu * PI * cs[0] * cs[1] * sn[2]; s[1][0] = s[0][1];
    s[0][2] = 2.0 * mu * PI * cs[0] * cs[2] * sn[1]; s[2][0] = s[0][2];
    s[1][2] = 2.0 * mu * PI * cs[1] * cs[2] * sn[0]; s[2][1] = s[1][2];
    for (int i = 0; i < 3; ++i)
        for (int j = 0; j < 3; ++j) r[i] = r[i] + s[i][j] * n[j];
}

__device__ inline void dev_analytic(int id, const double* sn, const double* cs, double r[3]) {
    const double PI = DATA_PI, SQ2 = 1.4142135623730951;
    if (id == LYMPH_FUN_IC_VELOCITY) {
        r[0] = SQ2 * PI * cs[0] * sn[1] * sn[2];
        r[1] = SQ2 * PI * sn[0] * cs[1] * sn[2];
        r[2] = SQ2 * PI * sn[0] * sn[1] * cs[2];
    } else if (id == LYMPH_FUN_UEX) {
        dev_u_space(sn, cs, r);
    } else {
        r[0] = r[1] = r[2] = 0.0;
    }
}

enum { VEC_RHS = 0, VEC_PROJECT = 1 };   // MAKE_RHS_FREE, L2 projection

struct VecArgs {
    const int32_t* poly_ptr;
    const int32_t* poly_tets;
    const int32_t* tet_mat;
    const int32_t* neigh;
    const int32_t* fun_tag;
    const double* mat;
    const double* fk;
    const double* jdet;
    const double* nrm;
    const double* area;
    const double* bbox;
    const double* hk;
    const RefTables* ref;
    double alpha, theta;
    int fid, did, nid;   // data function ids
    const double* R;     // modal factor (projection only)
    double scale;
    double* out;         // [n_poly][ND]
};

constexpr int VEC_THREADS = 128;   // k_damping

// Shape of k_vector per degree: T threads (the rows ND and the 3 R tasks per
// round of points fill them), R tabulated points at once.
template <int PD> struct VecShape {
    static constexpr int T = PD >= 3 ? 128 : (PD == 2 ? 96 : 32);
    static constexpr int R = PD == 4 ? 64 : Deg<PD>::NQ3;
    static_assert(R >= Deg<PD>::NQ2, "a face's points fit the table");
};

// solve_LU(R^T, R, b) (vet_mat_operations.f90:123-153) in the reference's
// operation order, one lane: forward substitution y_i = (b_i - sum_{j<i}
// R(j,i) y_j) / R(i,i), then back substitution x_i = (y_i - sum_{j>i} R(i,j)
// x_j) / R(i,i), both sums in increasing j.  Used by the set-up projection,
// where the solve sees the full coefficient vector and its rounding matters
// most; O(Np^2) sequential work once per polyhedron.
__device__ inline void lane_solve_rtr(int NP, const double* __restrict__ R, double* b) {
    for (int i = 0; i < NP; ++i) {
        double y = b[i];
        for (int j = 0; j < i; ++j) y = y - R[j * NP + i] * b[j];
        b[i] = y / R[i * NP + i];
    }
    for (int i = NP - 1; i >= 0; --i) {
        double x = b[i];
        for (int j = i + 1; j < NP; ++j) x = x - R[i * NP + j] * b[j];
        b[i] = x / R[i * NP + i];
    }
}

// MAKE_RHS_FREE (matrix_free.f90:467-843) with MAKE_RHS_VOLUME / MAKE_RHS_FACE
// (assemble_element.f90:171-390), or COMPUTE_MODAL_COEFFICIENTS_FREE
// (matrix_free.f90:847-997): one CTA per polyhedron.
//
// FP64-pipe bound: the sine and cosine of each quadrature coordinate, the
// Legendre values and the sums over the points.  So each coordinate of a point
// is one task (its interval map, every degree's value and its sine and cosine
// formed once), the weight is multiplied into the data once per point and
// component, and data functions that are zero everywhere (f_null,
// ic_displacement, uex_stat) do no quadrature.  Values and sums keep
// legendre_1d's and the reference's order: the projection's solve amplifies a
// change of rounding by the condition number of the mass matrix.
template <int PD, int MODE>
__global__ void __launch_bounds__(VecShape<PD>::T, PD < 3 ? 1 : (MODE == VEC_PROJECT ? 8 : 6)) k_vector(VecArgs A) {
    using D = Deg<PD>;
    constexpr int NP = D::NP, ND = D::ND, NQ3 = D::NQ3, NQ2 = D::NQ2, T = VecShape<PD>::T, R = VecShape<PD>::R, L1 = PD + 1;
    extern __shared__ double vsm[];
    double* s_acc = vsm;                  // [ND]
    double* s_phi = s_acc + ND;           // [R][NP]
    double* s_leg = s_phi + R * NP;       // [R][3][L1]
    double* s_sc = s_leg + R * 3 * L1;    // [R][3] sines, [R][3] cosines
    double* s_wd = s_sc + R * 6;          // [R][3] data (times weight in the volume)
    double* s_dphi = s_wd + R * 3;        // faces: [NQ2][3][NP]
    double* s_dleg = s_dphi + NQ2 * 3 * NP;   // faces: [NQ2][3][L1] derivatives
    __shared__ BoxC box;
    __shared__ DerTab<PD> der;
    const int tid = threadIdx.x, P = blockIdx.x;
    load_der<PD>(&der);
    if (tid < 3) box_consts(&A.bbox[P * 6], &box, tid);
    for (int i = tid; i < ND; i += T) s_acc[i] = 0.0;
    const bool vol = MODE == VEC_RHS ? A.fid != LYMPH_F_NULL
                                 : (A.fid == LYMPH_FUN_IC_VELOCITY || A.fid == LYMPH_FUN_UEX);
    const bool bnd = MODE == VEC_RHS && (A.did != LYMPH_GD_NULL || A.nid == LYMPH_GN);
    const int k1 = vol || bnd ? A.poly_ptr[P + 1] : A.poly_ptr[P];
    for (int kt = A.poly_ptr[P]; kt < k1; ++kt) {
        const int t = A.poly_tets[kt];
        const double* fk = &A.fk[t * 12];
        const int mid = A.tet_mat[t];
        const double rho = A.mat[mid * 3 + 0], lam = A.mat[mid * 3 + 1], mu = A.mat[mid * 3 + 2];
        const double aj = fabs(A.jdet[t]);
        // RHS: per-tetrahedron integral added to the polyhedron's vector
        // (MAKE_RHS_VOLUME then the row copy, matrix_free.f90:711-717);
        // projection: one running integral over all sub-tetrahedra
        // (uex_integral, matrix_free.f90:960-972)
        double s = 0.0;   // this thread's row (T >= ND)
        static_assert(T >= ND, "one thread per row");
        if (vol) {
            if (MODE != VEC_RHS && tid < ND) s = s_acc[tid];
            for (int q0 = 0; q0 < NQ3; q0 += R) {
                const int nq = (NQ3 - q0) < R ? (NQ3 - q0) : R;
                __syncthreads();
                for (int it = tid; it < nq * 3; it += T) {
                    const int qq = it / 3, d = it - qq * 3;
                    const double* nt = &A.ref->nodtet3[(q0 + qq) * 4];
                    double x = 0.0;
                    for (int l = 0; l < 4; ++l) x = x + fk[d * 4 + l] * nt[l];
                    legendre_vals<PD>(&box, d, x, s_leg + it * L1);
                    sincos(DATA_PI * x, &s_sc[it], &s_sc[R * 3 + it]);
                }
                __syncthreads();
                for (int qq = tid; qq < nq; qq += T) {
                    double r[3];
                    const double *sn = &s_sc[qq * 3], *cs = &s_sc[R * 3 + qq * 3];
                    if (MODE == VEC_RHS) dev_forcing(A.fid, lam, mu, rho, sn, cs, r);
                    else dev_analytic(A.fid, sn, cs, r);
                    const double w = aj * A.ref->weitet3[q0 + qq];
                    s_wd[qq * 3 + 0] = w * r[0]; s_wd[qq * 3 + 1] = w * r[1]; s_wd[qq * 3 + 2] = w * r[2];
                }
                for (int it = tid; it < nq * NP; it += T) {
                    const int q = it / NP, f = it - q * NP;
                    const double* tq = s_leg + q * 3 * L1;
                    s_phi[it] = tq[der.deg[f][0]] * tq[L1 + der.deg[f][1]] * tq[2 * L1 + der.deg[f][2]];
                }
                __syncthreads();
                if (tid < ND) {
                    const int i = tid / NP, m = tid - i * NP;
#pragma unroll 4
                    for (int q = 0; q < nq; ++q) s = s + s_wd[q * 3 + i] * s_phi[q * NP + m];
                }
            }
            if (tid < ND) {
                if (MODE == VEC_RHS) s_acc[tid] += s;
                else s_acc[tid] = s;
            }
        }
        // boundary faces of this tetrahedron (only boundary faces are added, :809-819)
        if constexpr (MODE == VEC_RHS)
        for (int f = 0; bnd && f < 4; ++f) {
            const int E2 = A.neigh[t * 4 + f];
            if (E2 != LYMPH_BC_DIRI && E2 != LYMPH_BC_NEUM) continue;
            if (E2 == LYMPH_BC_DIRI ? A.did == LYMPH_GD_NULL : A.nid != LYMPH_GN) continue;   // zero data
            const int tag = A.fun_tag ? A.fun_tag[t * 4 + f] : 1;
            const double nv[3] = {A.nrm[t * 12 + f * 3], A.nrm[t * 12 + f * 3 + 1], A.nrm[t * 12 + f * 3 + 2]};
            const double ar = A.area[t * 4 + f];
            __syncthreads();
            for (int it = tid; it < NQ2 * 3; it += T) {
                const int q = it / 3, j = it - q * 3;
                // the basis point (basis_boundary, basis_function.f90:560-577)
                const double* nt = &A.ref->nodtria2[q * 4];
                double x = 0.0;
                for (int l = 0; l < 4; ++l) x = x + face_map(fk, A.ref, f, j, l) * nt[l];
                double dv;
                for (int n = 0; n <= PD; ++n) {
                    legendre_1d(x, n, A.bbox[P * 6 + 2 * j], A.bbox[P * 6 + 2 * j + 1], &s_leg[it * L1 + n], &dv);
                    s_dleg[it * L1 + n] = dv;
                }
                // the data point as MAKE_RHS_FACE forms it (assemble_element.f90:313-320)
                const double* nm = &A.ref->node_maps[f * 16];
                double y = 0.0;
                for (int kk = 0; kk < 4; ++kk)
                    for (int tt = 0; tt < 4; ++tt) y = y + fk[j * 4 + kk] * nm[kk * 4 + tt] * nt[tt];
                sincos(DATA_PI * y, &s_sc[it], &s_sc[R * 3 + it]);
            }
            __syncthreads();
            for (int q = tid; q < NQ2; q += T) {
                double g[3];
                const double *sn = &s_sc[q * 3], *cs = &s_sc[R * 3 + q * 3];
                if (E2 == LYMPH_BC_DIRI) dev_dirichlet(A.did, tag, sn, cs, g);
                else dev_neumann(A.nid, lam, mu, nv, tag, sn, cs, g);
                s_wd[q * 3 + 0] = g[0]; s_wd[q * 3 + 1] = g[1]; s_wd[q * 3 + 2] = g[2];
            }
            for (int it = tid; it < NQ2 * NP; it += T) {
                const int q = it / NP, fb = it - q * NP;
                const double *tv = s_leg + q * 3 * L1, *td = s_dleg + q * 3 * L1;
                const int bx = der.deg[fb][0], by = L1 + der.deg[fb][1], bz = 2 * L1 + der.deg[fb][2];
                const double vx = tv[bx], vy = tv[by], vz = tv[bz];
                s_phi[it] = vx * vy * vz;
                s_dphi[(q * 3 + 0) * NP + fb] = td[bx] * vy * vz;
                s_dphi[(q * 3 + 1) * NP + fb] = vx * td[by] * vz;
                s_dphi[(q * 3 + 2) * NP + fb] = vx * vy * td[bz];
            }
            __syncthreads();
            const double sigma = A.alpha * (double)(PD * PD) / A.hk[P] * (lam + 2 * mu);
            const double n0 = nv[0], n1 = nv[1], n2 = nv[2];
            const double a0 = fabs(n0) * fabs(n0), a1 = fabs(n1) * fabs(n1), a2 = fabs(n2) * fabs(n2);
            for (int r = tid; r < ND; r += T) {
                const int i = r / NP, m = r % NP;
                double rf = 0.0;
                for (int q = 0; q < NQ2; ++q) {
                    const double w = A.ref->weitria2[q];
                    const double* gd = &s_wd[q * 3];
                    const double ph = s_phi[q * NP + m];
                    if (E2 == LYMPH_BC_DIRI) {
                        const double g0 = s_dphi[(q * 3 + 0) * NP + m], g1 = s_dphi[(q * 3 + 1) * NP + m],
                                     g2 = s_dphi[(q * 3 + 2) * NP + m];
                        double tv, sv;
                        if (i == 0) {
                            tv = (lam + 2 * mu) * g0 * gd[0] * n0 + mu * g1 * gd[0] * n1 + mu * g2 * gd[0] * n2 +
                                 lam * g0 * gd[1] * n1 + mu * g1 * gd[1] * n0 + lam * g0 * gd[2] * n2 + mu * g2 * gd[2] * n0;
                            sv = ph * gd[0] * (a0 + 0.5 * a1 + 0.5 * a2) + 0.5 * ph * gd[1] * n0 * n1 + 0.5 * ph * gd[2] * n0 * n2;
                        } else if (i == 1) {
                            tv = (lam + 2 * mu) * g1 * gd[1] * n1 + mu * g0 * gd[1] * n0 + mu * g2 * gd[1] * n2 +
                                 lam * g1 * gd[0] * n0 + mu * g0 * gd[0] * n1 + lam * g1 * gd[2] * n2 + mu * g2 * gd[2] * n1;
                            sv = ph * gd[1] * (a1 + 0.5 * a0 + 0.5 * a2) + 0.5 * ph * gd[0] * n0 * n1 + 0.5 * ph * gd[2] * n1 * n2;
                        } else {
                            tv = (lam + 2 * mu) * g2 * gd[2] * n2 + mu * g0 * gd[2] * n0 + mu * g1 * gd[2] * n1 +
                                 lam * g2 * gd[0] * n0 + mu * g0 * gd[0] * n2 + lam * g2 * gd[1] * n1 + mu * g1 * gd[1] * n2;
                            sv = ph * gd[2] * (a2 + 0.5 * a0 + 0.5 * a1) + 0.5 * ph * gd[0] * n0 * n2 + 0.5 * ph * gd[1] * n1 * n2;
                        }
                        rf = rf + A.theta * w * tv * ar + sigma * w * sv * ar;
                    } else {
                        rf = rf + w * ph * gd[i] * ar;
                    }
                }
                if (rf != 0.0) s_acc[r] += rf;
            }
        }
    }
    __syncthreads();
    if (MODE == VEC_RHS) {
        for (int r = tid; r < ND; r += T) A.out[(int64_t)P * ND + r] = s_acc[r];
        return;
    }
    // L2 projection: solve_LU(R^T, R) per component with the modal factor
    if (vol && tid < 3) lane_solve_rtr(NP, A.R + (int64_t)P * NP * NP, &s_acc[tid * NP]);
    __syncthreads();
    for (int r = tid; r < ND; r += T) A.out[(int64_t)P * ND + r] = s_acc[r] * A.scale;
}

// MAKE_DAMPING_FACE (assemble_element.f90:666-731) summed over the absorbing
// faces of each polyhedron that has some: one CTA per such polyhedron, the
// face's quadrature points and P's basis values in shared memory, each thread
// owning fixed entries of the ND x ND block D (row (i, m), column (j, n)):
//   D += |face| w_q (phi_m phi_n) C_ij,
//   C = c_t (t1 t1^T + t2 t2^T) + c_n n n^T = c_t (I - n n^T) + c_n n n^T,
// c_t = sqrt(rho mu), c_n = sqrt(rho (lambda + 2 mu)) of the face's
// tetrahedron.  phi_m phi_n is formed before the weight, so D is exactly
// symmetric.
template <int PD>
__global__ void __launch_bounds__(VEC_THREADS) k_damping(const int32_t* __restrict__ abs_poly,
                                                       const int32_t* __restrict__ abs_ptr,
                                                       const int32_t* __restrict__ abs_faces, const double* __restrict__ fk,
                                                       const double* __restrict__ nrm, const double* __restrict__ area,
                                                       const double* __restrict__ bbox, const int32_t* __restrict__ tet_mat,
                                                       const double* __restrict__ mat, const RefTables* __restrict__ ref,
                                                       double* __restrict__ D) {
    using Dg = Deg<PD>;
    constexpr int NP = Dg::NP, ND = Dg::ND, NQ2 = Dg::NQ2;
    __shared__ double s_phi[NQ2 * NP];
    __shared__ double s_pt[NQ2 * 3];
    const int a = blockIdx.x, tid = threadIdx.x, P = abs_poly[a];
    const double* bb = &bbox[P * 6];
    double* Da = D + (int64_t)a * ND * ND;
    for (int e = tid; e < ND * ND; e += VEC_THREADS) Da[e] = 0.0;
    for (int k = abs_ptr[a]; k < abs_ptr[a + 1]; ++k) {
        const int code = abs_faces[k], t = code >> 2, f = code & 3;
        __syncthreads();
        for (int q = tid; q < NQ2; q += VEC_THREADS) face_point(&fk[t * 12], ref, f, q, &s_pt[q * 3]);
        __syncthreads();
        for (int it = tid; it < NQ2 * NP; it += VEC_THREADS) {
            const int q = it / NP, fb = it % NP;
            double dp[3];
            basis_eval(&s_pt[q * 3], bb, &ref->blist[fb * 3], &s_phi[q * NP + fb], dp);
        }
        __syncthreads();
        const double* n = &nrm[t * 12 + f * 3];
        const int mid = tet_mat[t];
        const double rho = mat[mid * 3 + 0], lam = mat[mid * 3 + 1], mu = mat[mid * 3 + 2];
        const double ct = sqrt(rho * mu), cn = sqrt(rho * (lam + 2.0 * mu));
        const double ar = area[t * 4 + f];
        for (int e = tid; e < ND * ND; e += VEC_THREADS) {
            const int r = e / ND, cc = e - r * ND;
            const int i = r / NP, m = r - i * NP, j = cc / NP, nn = cc - j * NP;
            const double nij = n[i] * n[j];
            const double C = ct * ((i == j ? 1.0 : 0.0) - nij) + cn * nij;
            double s = 0.0;
            for (int q = 0; q < NQ2; ++q) s = s + ref->weitria2[q] * (s_phi[q * NP + m] * s_phi[q * NP + nn]);
            Da[e] += ar * C * s;
        }
    }
}

// W = M (x) I + dt/2 D for each polyhedron with absorbing faces (M: the
// rho-weighted mass matrix M_loc of the polyhedron, the same for each
// component).
__global__ void k_damping_w(int n_abs, int NP, const int32_t* __restrict__ abs_poly, const double* __restrict__ M,
                            const double* __restrict__ D, double half_dt, double* __restrict__ W) {
    const int ND = 3 * NP;
    const int64_t total = (int64_t)n_abs * ND * ND;
    for (int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < total; e += (int64_t)gridDim.x * blockDim.x) {
        const int64_t a = e / ((int64_t)ND * ND);
        const int rc = (int)(e - a * ND * ND), r = rc / ND, cc = rc - r * ND;
        const int i = r / NP, m = r - i * NP, j = cc / NP, nn = cc - j * NP;
        const double mv = (i == j) ? M[(int64_t)abs_poly[a] * NP * NP + m * NP + nn] : 0.0;
        W[e] = mv + half_dt * D[e];
    }
}

// Point source: rhs[P][i*Np + m] = dir_i phi_m(x0) for the polyhedron P
// that contains x0 (one block of Np threads); the rest of rhs was zeroed by
// the caller.  The spatial part of a Ricker source f = dir delta(x - x0) R(t),
// whose time part R(t) enters through the time-function values.
__global__ void k_point_source(int Np, int P, const double* __restrict__ bbox, const RefTables* __restrict__ ref,
                               double x, double y, double z, double dx, double dy, double dz, double* rhs) {
    const int m = threadIdx.x;
    if (m >= Np) return;
    const double pt[3] = {x, y, z};
    double ph, dp[3];
    basis_eval(pt, &bbox[P * 6], &ref->blist[m * 3], &ph, dp);
    const int64_t base = (int64_t)P * 3 * Np;
    rhs[base + 0 * Np + m] = dx * ph;
    rhs[base + 1 * Np + m] = dy * ph;
    rhs[base + 2 * Np + m] = dz * ph;
}

// Double-couple source on tetrahedron t of polyhedron P (one block of Np
// threads, thread m): rhs[P][(i, m)] += sum_q w_q |J| sum_j moment(i, j)
// dphi_j(m, x_q), the body of MAKE_DOUBLE_COUPLE
// (assemble_element.f90:116-167) with the moment density
// (s n^T + n s^T) M0 / V of problem_data_and_properties.f90:317-335, in the
// reference's order (q outer, j inner).
__global__ void k_double_couple(int Np, int nq3, int t, int P, const double* __restrict__ fk,
                                const double* __restrict__ jdet, const double* __restrict__ bbox,
                                const RefTables* __restrict__ ref, const double* __restrict__ moment, double* rhs) {
    const int m = threadIdx.x;
    if (m >= Np) return;
    const double* F = fk + (int64_t)t * 12;
    const double aj = fabs(jdet[t]);
    double acc[3] = {0.0, 0.0, 0.0};
    for (int q = 0; q < nq3; ++q) {
        const double* nq = &ref->nodtet3[q * 4];
        double pt[3];
        for (int a = 0; a < 3; ++a) pt[a] = F[a * 4 + 0] * nq[0] + F[a * 4 + 1] * nq[1] + F[a * 4 + 2] * nq[2] + F[a * 4 + 3];
        double ph, dp[3];
        basis_eval(pt, &bbox[P * 6], &ref->blist[m * 3], &ph, dp);
        for (int i = 0; i < 3; ++i) {
            double reduct = 0.0;
            for (int j = 0; j < 3; ++j) reduct = reduct + moment[i * 3 + j] * dp[j];
            acc[i] = acc[i] + ref->weitet3[q] * aj * reduct;
        }
    }
    const int64_t base = (int64_t)P * 3 * Np;
    for (int i = 0; i < 3; ++i) rhs[base + i * Np + m] += acc[i];
}

template <int PD, int WHICH>
int launch_assemble(lymph_ctx* c, double* out, bool write_mass) {
    AsmArgs A;
    A.row_ptr = c->d_row_ptr; A.blk_row = c->d_blk_row; A.col = c->d_col; A.bf_ptr = c->d_bf_ptr; A.bf = c->d_bf;
    A.poly_ptr = c->d_poly_ptr; A.poly_tets = c->d_poly_tets; A.tet_poly = c->d_tet_poly; A.tet_mat = c->d_tet_mat;
    A.neigh = c->d_neigh; A.mat = c->d_mat; A.fk = c->d_fk; A.jdet = c->d_jdet; A.nrm = c->d_normal; A.area = c->d_area;
    A.bbox = c->d_bbox; A.hk = c->d_hk; A.ref = c->d_ref; A.alpha = c->alpha; A.theta = c->theta; A.out = out;
    A.M = write_mass ? c->d_M : nullptr; A.Mm = write_mass ? c->d_Mm : nullptr;
    A.block0 = 0;
    const size_t sself = asm_self_smem<PD, WHICH>();
    LYMPH_CUDA_TRY(cudaFuncSetAttribute(k_assemble_self<PD, WHICH>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sself));
    k_assemble_self<PD, WHICH><<<c->n_poly, AsmShape<PD>::T, sself, c->stream>>>(A);
    c->launches++;
    LYMPH_CUDA_TRY(cudaGetLastError());
    if constexpr (WHICH != ASM_MASS) {
        const size_t snb = asm_nb_smem<PD, WHICH>();
        LYMPH_CUDA_TRY(cudaFuncSetAttribute(k_assemble_nb<PD, WHICH>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)snb));
        const int64_t chunk = 1 << 20;
        for (int64_t b0 = 0; b0 < c->n_blocks; b0 += chunk) {
            A.block0 = b0;
            const int64_t nb = c->n_blocks - b0 < chunk ? c->n_blocks - b0 : chunk;
            k_assemble_nb<PD, WHICH><<<(unsigned)nb, AsmShape<PD>::TN, snb, c->stream>>>(A);
            c->launches++;
            LYMPH_CUDA_TRY(cudaGetLastError());
        }
    }
    return LYMPH_OK;
}

template <int WHICH>
int assemble_degree(lymph_ctx* c, double* out, bool write_mass) {
    switch (c->p) {
        case 1: return launch_assemble<1, WHICH>(c, out, write_mass);
        case 2: return launch_assemble<2, WHICH>(c, out, write_mass);
        case 3: return launch_assemble<3, WHICH>(c, out, write_mass);
        case 4: return launch_assemble<4, WHICH>(c, out, write_mass);
        default: lymph_set_error("degree not supported on the device"); return LYMPH_ERR_INVALID;
    }
}

template <int PD, int MODE>
int launch_vector(lymph_ctx* c, int fid, int did, int nid, double scale, double* out) {
    VecArgs A;
    A.poly_ptr = c->d_poly_ptr; A.poly_tets = c->d_poly_tets; A.tet_mat = c->d_tet_mat; A.neigh = c->d_neigh;
    A.fun_tag = c->d_fun_tag; A.mat = c->d_mat; A.fk = c->d_fk; A.jdet = c->d_jdet; A.nrm = c->d_normal;
    A.area = c->d_area; A.bbox = c->d_bbox; A.hk = c->d_hk; A.ref = c->d_ref; A.alpha = c->alpha; A.theta = c->theta;
    A.fid = fid; A.did = did; A.nid = nid; A.R = c->d_Rm; A.scale = scale; A.out = out;
    using D = Deg<PD>;
    using V = VecShape<PD>;
    const size_t face = (size_t)D::NQ2 * 3 * (D::NP + PD + 1);   // gradient tables of a boundary face (RHS only)
    const size_t smem = sizeof(double) * ((size_t)D::ND + (size_t)V::R * (D::NP + 3 * (PD + 1) + 9) + (MODE == VEC_RHS ? face : 0));
    LYMPH_CUDA_TRY(cudaFuncSetAttribute(k_vector<PD, MODE>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    k_vector<PD, MODE><<<c->n_poly, V::T, smem, c->stream>>>(A);
    c->launches++;
    LYMPH_CUDA_TRY(cudaGetLastError());
    return LYMPH_OK;
}

}  // namespace

// ---------------------------------------------------------------------------
// host entry points used by abi.cu
// ---------------------------------------------------------------------------
int lymph_dev_geometry(lymph_ctx* c) {
    if (c->n_tet > 0) {
        k_geometry<<<(c->n_tet + 127) / 128, 128, 0, c->stream>>>(c->n_tet, c->d_coords, c->d_tet_vert, c->d_fk,
                                                                 c->d_jdet, c->d_normal, c->d_area, c->d_status);
        c->launches++;
        LYMPH_CUDA_TRY(cudaGetLastError());
    }
    if (c->n_poly > 0) {
        k_bbox<<<(c->n_poly + BBOX_WARPS - 1) / BBOX_WARPS, 32 * BBOX_WARPS, 0, c->stream>>>(c->n_poly, c->d_poly_ptr, c->d_poly_tets, c->d_tet_vert,
                                                              c->d_coords, c->d_bbox, c->d_hk);
        c->launches++;
        LYMPH_CUDA_TRY(cudaGetLastError());
    }
    return LYMPH_OK;
}

// The rho-weighted and the plain mass matrix of every polyhedron (what the
// mixed operators need of the FP64 assembly).
int lymph_dev_mass(lymph_ctx* c) { return assemble_degree<ASM_MASS>(c, nullptr, true); }

// Every FP64 block of the operator (LYMPH_BLOCKS_K) or of the DG norm
// (LYMPH_BLOCKS_ADG) into out; with write_mass also the mass matrices.
int lymph_dev_assemble(lymph_ctx* c, int which, double* out, bool write_mass) {
    return which == LYMPH_BLOCKS_ADG ? assemble_degree<ASM_ADG>(c, out, write_mass) : assemble_degree<ASM_K>(c, out, write_mass);
}

int lymph_dev_cholesky(lymph_ctx* c) {
    const int warps_per_block = 4;
    size_t smem = sizeof(double) * warps_per_block * c->Np * c->Np;
    unsigned grid = (unsigned)((c->n_poly + warps_per_block - 1) / warps_per_block);
    k_cholesky<<<grid, 32 * warps_per_block, smem, c->stream>>>(c->n_poly, c->Np, c->d_M, c->d_R, c->d_status);
    k_cholesky<<<grid, 32 * warps_per_block, smem, c->stream>>>(c->n_poly, c->Np, c->d_Mm, c->d_Rm, c->d_status);
    const size_t smem_inv = sizeof(double) * 2 * INV_MATS * c->Np * c->Np;
    // raise (never lower) the dynamic shared-memory limit: other contexts may launch with a larger Np
    LYMPH_CUDA_TRY(cudaFuncSetAttribute(k_mass_inverse, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                        (int)(sizeof(double) * 2 * INV_MATS * MAX_NP * MAX_NP)));
    k_mass_inverse<<<(c->n_poly + INV_MATS - 1) / INV_MATS, INV_THREADS, smem_inv, c->stream>>>(c->n_poly, c->Np, c->d_R, c->d_Minv);
    c->launches += 3;
    LYMPH_CUDA_TRY(cudaGetLastError());
    return LYMPH_OK;
}

// The damping blocks of the absorbing faces (once per assembly) and the
// inverses of M (x) I + dt/2 D for the context's dt: W, its Cholesky factor
// (cholesky, one warp per polyhedron) and the explicit column-major inverse
// (solve_LU per column), as for the mass matrix.
int lymph_dev_damping(lymph_ctx* c, bool assemble) {
    if (c->n_abs <= 0) return LYMPH_OK;
    const int ND = c->nd;
    if (assemble) {
        switch (c->p) {
            case 1: k_damping<1><<<c->n_abs, VEC_THREADS, 0, c->stream>>>(c->d_abs_poly, c->d_abs_ptr, c->d_abs_faces, c->d_fk, c->d_normal, c->d_area, c->d_bbox, c->d_tet_mat, c->d_mat, c->d_ref, c->d_Dabs); break;
            case 2: k_damping<2><<<c->n_abs, VEC_THREADS, 0, c->stream>>>(c->d_abs_poly, c->d_abs_ptr, c->d_abs_faces, c->d_fk, c->d_normal, c->d_area, c->d_bbox, c->d_tet_mat, c->d_mat, c->d_ref, c->d_Dabs); break;
            case 3: k_damping<3><<<c->n_abs, VEC_THREADS, 0, c->stream>>>(c->d_abs_poly, c->d_abs_ptr, c->d_abs_faces, c->d_fk, c->d_normal, c->d_area, c->d_bbox, c->d_tet_mat, c->d_mat, c->d_ref, c->d_Dabs); break;
            case 4: k_damping<4><<<c->n_abs, VEC_THREADS, 0, c->stream>>>(c->d_abs_poly, c->d_abs_ptr, c->d_abs_faces, c->d_fk, c->d_normal, c->d_area, c->d_bbox, c->d_tet_mat, c->d_mat, c->d_ref, c->d_Dabs); break;
            default: lymph_set_error("degree not supported on the device"); return LYMPH_ERR_INVALID;
        }
        c->launches++;
        LYMPH_CUDA_TRY(cudaGetLastError());
    }
    const int64_t total = (int64_t)c->n_abs * ND * ND;
    const unsigned gw = (unsigned)((total + 255) / 256 < 4096 ? (total + 255) / 256 : 4096);
    k_damping_w<<<gw, 256, 0, c->stream>>>(c->n_abs, c->Np, c->d_abs_poly, c->d_M, c->d_Dabs, 0.5 * c->dt, c->d_Wabs);
    const size_t smem = sizeof(double) * (size_t)ND * ND;  // one warp per block: its ND x ND factor
    // raise (never lower) k_cholesky's dynamic shared-memory limit: the mass
    // factorisation launches it with up to 4 Np^2 doubles per block
    const size_t lim = smem > (size_t)48 * 1024 ? smem : (size_t)48 * 1024;
    LYMPH_CUDA_TRY(cudaFuncSetAttribute(k_cholesky, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)lim));
    k_cholesky<<<c->n_abs, 32, smem, c->stream>>>(c->n_abs, ND, c->d_Wabs, c->d_Rw, c->d_status);
    k_inverse_columns<<<(unsigned)((c->n_abs + 3) / 4), 128, 0, c->stream>>>(c->n_abs, ND, c->d_Rw, c->d_Winv);
    c->launches += 3;
    c->winv_dt = c->dt;
    LYMPH_CUDA_TRY(cudaGetLastError());
    return LYMPH_OK;
}

int lymph_dev_point_source(lymph_ctx* c, int P, const double x0[3], const double dir[3], double* out) {
    LYMPH_CUDA_TRY(cudaMemsetAsync(out, 0, sizeof(double) * (size_t)c->n_poly * c->nd, c->stream));
    k_point_source<<<1, 64, 0, c->stream>>>(c->Np, P, c->d_bbox, c->d_ref, x0[0], x0[1], x0[2], dir[0], dir[1], dir[2], out);
    c->launches++;
    LYMPH_CUDA_TRY(cudaGetLastError());
    return LYMPH_OK;
}

int lymph_dev_double_couple(lymph_ctx* c, int t, int P, const double moment[9], double* out) {
    double* d_m = nullptr;
    LYMPH_CUDA_TRY(cudaMalloc(&d_m, sizeof(double) * 9));
    cudaError_t e = cudaMemcpyAsync(d_m, moment, sizeof(double) * 9, cudaMemcpyHostToDevice, c->stream);
    if (e == cudaSuccess) {
        k_double_couple<<<1, 64, 0, c->stream>>>(c->Np, c->nq3, t, P, c->d_fk, c->d_jdet, c->d_bbox, c->d_ref, d_m, out);
        c->launches++;
        e = cudaGetLastError();
    }
    if (e == cudaSuccess) e = cudaStreamSynchronize(c->stream);
    cudaFree(d_m);
    if (e != cudaSuccess) {
        lymph_set_error(std::string("lymph_dev_double_couple: ") + cudaGetErrorString(e));
        return LYMPH_ERR_CUDA;
    }
    return LYMPH_OK;
}

int lymph_dev_vector(lymph_ctx* c, int mode, int fid, int did, int nid, double scale, double* out) {
    switch (c->p) {
        case 1: return mode == VEC_RHS ? launch_vector<1, VEC_RHS>(c, fid, did, nid, scale, out)
                                       : launch_vector<1, VEC_PROJECT>(c, fid, did, nid, scale, out);
        case 2: return mode == VEC_RHS ? launch_vector<2, VEC_RHS>(c, fid, did, nid, scale, out)
                                       : launch_vector<2, VEC_PROJECT>(c, fid, did, nid, scale, out);
        case 3: return mode == VEC_RHS ? launch_vector<3, VEC_RHS>(c, fid, did, nid, scale, out)
                                       : launch_vector<3, VEC_PROJECT>(c, fid, did, nid, scale, out);
        case 4: return mode == VEC_RHS ? launch_vector<4, VEC_RHS>(c, fid, did, nid, scale, out)
                                       : launch_vector<4, VEC_PROJECT>(c, fid, did, nid, scale, out);
        default: lymph_set_error("degree not supported on the device"); return LYMPH_ERR_INVALID;
    }
}
