// step.cu -- the per-step hot kernel and the error norms.
//
// One CTA per polyhedron P fuses what TIME_STEP_MATRIX_FREE
// (src/matrix_free.f90:1230-1385) does for one element:
//   1. y = sum_b K_{P,col(b)} u_{col(b)}     (self + neighbour blocks; the
//      neighbour coefficients the reference receives by MPI_EXCHANGE_DOF are
//      gathered from global memory, L2-resident)
//   2. tmp = -y + F_stat + F_dyn g(t)
//   3. x = M^-1 tmp per component: the value of the reference's
//      solve_LU(R^T, R, tmp) (vet_mat_operations.f90:123-153), applied as a
//      dense FP64 product with the inverse built once from the same factor
//   4. u^{n+1} = dt^2 x + 2 u^n - u^{n-1}    (written over u^{n-1} in place)
// Blocks are stored column-major so that thread r (row r) reads
// K[c][r] for consecutive r: coalesced, streamed once per step with an
// evict-first hint so the state vectors stay in L2.  Threads are laid out as
// S column slices x ND rows, S chosen per degree so that ND*S fills whole
// warps; the S partial sums of a row are combined in a fixed order.

#include "step_body.cuh"

namespace {

using namespace stepk;

// One CTA per polyhedron.  Without the code of absorbing faces (ABS) p = 1 takes 32 registers
// instead of 38 with FP32 blocks, so 21 CTAs fit an SM instead of 17: 48 steps of 46,861
// polyhedra 5.08 -> 4.42 ms, of 3,013 466 -> 430 us; the bound of 20 holds every mode to
// that (30 products of the power iteration 8.89 -> 8.34 ms).  The integer columns of p = 2 keep few values
// per thread and wait for their loads: 8 CTAs per SM (32 registers) instead of 6 take
// 46,861 polyhedra from 46.2 to 37.8 ms, 737 from 0.89 to 0.87 (45.7 and 1.02 with FP64 products).
// The FP64 products of p = 2 load two blocks at once (8,000 hexahedra 5.47 -> 5.42 ms, 2,197
// 1.65 -> 1.62): left to itself the compiler loads one once the damping's code is gone.
// At p = 3 in FP64 6 CTAs' arrays of 20,752 bytes just fill the 132 KB division of an SM's
// memory; with 1,600 bytes more each the next larger one is taken and meshes of 1 to 3
// waves gain (1,296 tetrahedra 2.09 -> 2.01 ms, 1,331 hexahedra 2.62 -> 2.53; larger ones 0-1 %).
constexpr size_t step_pad(int p, bool ints) { return p == 3 && ints ? 1600 : 0; }
template <int PD, typename KT, int MODE, bool INT, bool ABS>
__global__ void __launch_bounds__(Shape<PD>::T, PD == 1 && sizeof(KT) == 4 ? 20 : (PD == 2 && INT ? 8 : Shape<PD>::MINB)) k_step(StepArgs A) {
    __shared__ __align__(16) char smem[SmemSize<PD, KT, Shape<PD>::S, INT>::bytes + step_pad(PD, INT)];
    step_poly<PD, KT, MODE, Shape<PD>::S, INT, false, ABS, PD == 3 ? 8 : 16, PD == 2 && sizeof(KT) == 8 && !INT ? 2 : 0>(A, blockIdx.x, smem);
}

// The same for at most one polyhedron per SM without absorbing faces, p <= 3.
template <int PD, typename KT, bool INT = int_columns(PD, sizeof(KT))>
__global__ void __launch_bounds__(Shape<PD>::T, 2) k_step_small(StepArgs A) {
    __shared__ __align__(16) char smem[SmemSize<PD, KT, Shape<PD>::S, INT>::bytes];
    extern __shared__ __align__(16) char dyn[];
    step_poly<PD, KT, MODE_STEP, Shape<PD>::S, INT, true>(A, blockIdx.x, smem, dyn);
}

__global__ void k_bump(int64_t* idx, int n) { *idx += n; }

// COMPUTE_ERROR_L2_MATRIX_FREE body per polyhedron: sum_i du_i^T M du_i.
__global__ void __launch_bounds__(L2_THREADS) k_l2_partial(int n_poly, int NP, const double* __restrict__ Mm,
                                                           const double* __restrict__ uh, const double* __restrict__ uex,
                                                           double* partial) {
    l2_partials(n_poly, NP, Mm, uh, uex, partial);
}
void launch_l2(lymph_ctx* c, const double* M, const double* uh, const double* uex) {
    k_l2_partial<<<l2_grid(c->n_poly, c->Np), L2_THREADS, 0, c->stream>>>(c->n_poly, c->Np, M, uh, uex, c->d_partial);
}

// ---- COMPUTE_ERROR_DG_MATRIX_FREE ----

struct DgArgs {
    const int32_t* row_ptr;
    const int64_t* bf_ptr;
    const int32_t* bf;
    const int32_t* poly_ptr;
    const int32_t* poly_tets;
    const int32_t* tet_poly;
    const int32_t* tet_mat;
    const int32_t* neigh;
    const double *mat, *fk, *jdet, *nrm, *area, *bbox, *hk;
    const RefTables* ref;
    const double *uh, *uex;
    double alpha;
    double* partial;   // [n_poly]
};

// Position of basis function (a, b, c) in the reference's order.
template <int PD> struct BasisPos {
    int i[PD + 1][PD + 1][PD + 1];
    constexpr BasisPos() : i() {
        constexpr Blist<PD> BL{};
        for (int k = 0; k < Deg<PD>::NP; ++k) i[BL.d[k][0]][BL.d[k][1]][BL.d[k][2]] = k;
    }
};

// Legendre polynomials and derivatives of degrees 0..PD at x (recurrences).
template <int PD> __device__ __forceinline__ void legendre_rec(double x, double* L, double* dL) {
    L[0] = 1.0;
    dL[0] = 0.0;
    L[1] = x;
    dL[1] = 1.0;
#pragma unroll
    for (int n = 1; n < PD; ++n) {
        L[n + 1] = ((2 * n + 1) * x * L[n] - n * L[n - 1]) * (1.0 / (n + 1));
        dL[n + 1] = dL[n - 1] + (2 * n + 1) * L[n];
    }
}

// The three components of sum_m u_m phi_m at a point, unscaled, by sum
// factorisation over the degree triples; at(m, j): coefficient m of component j.
template <int PD, typename At>
__device__ __forceinline__ void field_sf(At at, const double* X, const double* Y, const double* Z, double (&v)[3]) {
    constexpr BasisPos<PD> BP{};
    v[0] = v[1] = v[2] = 0.0;
#pragma unroll
    for (int a = 0; a <= PD; ++a) {
        double r[3] = {0.0, 0.0, 0.0};
#pragma unroll
        for (int b = 0; b <= PD - a; ++b) {
            double w[3] = {0.0, 0.0, 0.0};
#pragma unroll
            for (int c = 0; c <= PD - a - b; ++c)
#pragma unroll
                for (int j = 0; j < 3; ++j) w[j] = fma(at(BP.i[a][b][c], j), Z[c], w[j]);
#pragma unroll
            for (int j = 0; j < 3; ++j) r[j] = fma(w[j], Y[b], r[j]);
        }
#pragma unroll
        for (int j = 0; j < 3; ++j) v[j] = fma(r[j], X[a], v[j]);
    }
}

constexpr int DG_THREADS = 128;

// du_P . (A_PP du_P + sum_Q A_PQ du_Q), du = uh - uex, of the DG-norm blocks
// the reference assembles (strain energy of P's tetrahedra, penalty of the
// jumps on its faces), straight from the quadrature: a thread per point
// evaluates the gradient (volume) or the two sides' values (faces) of du by
// sum factorisation,
//     sum_q w (lambda (tr g)^2 + mu g : (g + g^T)) + sum_q W sigma v_P . T (v_P - v_Q),
// T z = n (n . z) / 2 + |n|^2 z / 2 and v_Q = 0 on a Dirichlet face.  FP64-pipe
// bound.  No block is formed: a tetrahedron costs (p+1)^3 evaluations instead
// of Np^2 moments per point, and no operator-sized buffer is needed.
template <int PD>
__global__ void __launch_bounds__(DG_THREADS, 4) k_dg_partial(const __grid_constant__ DgArgs A) {
    constexpr int NP = Deg<PD>::NP, ND = Deg<PD>::ND, NQ3 = (PD + 1) * (PD + 1) * (PD + 1), NQ2 = (PD + 1) * (PD + 1);
    constexpr BasisPos<PD> BP{};
    __shared__ double s_du[ND], s_red[DG_THREADS / 32];
    const int tid = threadIdx.x, P = blockIdx.x;
    for (int i = tid; i < ND; i += DG_THREADS) s_du[i] = A.uh[(int64_t)P * ND + i] - A.uex[(int64_t)P * ND + i];
    double mid[3], ih[3], hp = 1.0;
#pragma unroll
    for (int d = 0; d < 3; ++d) {
        const double lo = A.bbox[P * 6 + 2 * d], hi = A.bbox[P * 6 + 2 * d + 1];
        mid[d] = 0.5 * (lo + hi);
        ih[d] = 2.0 / (hi - lo);
        hp *= ih[d];
    }
    const double sc = sqrt(hp);   // phi = sc L_a L_b L_c
    __syncthreads();
    const int p0 = A.poly_ptr[P], n_vol = (A.poly_ptr[P + 1] - p0) * NQ3;
    double acc = 0.0;
    for (int it = tid; it < n_vol; it += DG_THREADS) {
        // the coefficients are read from shared memory at each point: hoisted
        // out of the loop, all 3 Np of them spill
        asm volatile("" ::: "memory");
        const int kt = it / NQ3, q = it - kt * NQ3, t = A.poly_tets[p0 + kt];
        const double* fk = &A.fk[(int64_t)t * 12];
        const double* nt = &A.ref->nodtet3[q * 4];
        double L[3][PD + 1], dL[3][PD + 1];
#pragma unroll
        for (int d = 0; d < 3; ++d) {
            const double x = fma(fk[d * 4], nt[0], fma(fk[d * 4 + 1], nt[1], fma(fk[d * 4 + 2], nt[2], fk[d * 4 + 3])));
            legendre_rec<PD>((x - mid[d]) * ih[d], L[d], dL[d]);
        }
        double g[3][3] = {};   // g[k][j] = d_k du_j
#pragma unroll
        for (int a = 0; a <= PD; ++a) {
            double r0[3] = {}, r1[3] = {}, r2[3] = {};
#pragma unroll
            for (int b = 0; b <= PD - a; ++b) {
                double w0[3] = {}, w1[3] = {};
#pragma unroll
                for (int c = 0; c <= PD - a - b; ++c)
#pragma unroll
                    for (int j = 0; j < 3; ++j) {
                        const double u = s_du[j * NP + BP.i[a][b][c]];
                        w0[j] = fma(u, L[2][c], w0[j]);
                        w1[j] = fma(u, dL[2][c], w1[j]);
                    }
#pragma unroll
                for (int j = 0; j < 3; ++j) {
                    r0[j] = fma(w0[j], L[1][b], r0[j]);
                    r1[j] = fma(w0[j], dL[1][b], r1[j]);
                    r2[j] = fma(w1[j], L[1][b], r2[j]);
                }
            }
#pragma unroll
            for (int j = 0; j < 3; ++j) {
                g[0][j] = fma(r0[j], dL[0][a], g[0][j]);
                g[1][j] = fma(r1[j], L[0][a], g[1][j]);
                g[2][j] = fma(r2[j], L[0][a], g[2][j]);
            }
        }
#pragma unroll
        for (int k = 0; k < 3; ++k)
#pragma unroll
            for (int j = 0; j < 3; ++j) g[k][j] *= sc * ih[k];
        const int m = A.tet_mat[t];
        const double tr = g[0][0] + g[1][1] + g[2][2];
        double gg = 0.0;
#pragma unroll
        for (int k = 0; k < 3; ++k)
#pragma unroll
            for (int j = 0; j < 3; ++j) gg = fma(g[k][j], g[k][j] + g[j][k], gg);
        acc = fma(A.ref->weitet3[q] * fabs(A.jdet[t]), A.mat[m * 3 + 1] * (tr * tr) + A.mat[m * 3 + 2] * gg, acc);
    }
    // faces that carry a term: the self block's list, first in P's row
    const int64_t e0 = A.bf_ptr[A.row_ptr[P]];
    const int n_face = (int)(A.bf_ptr[A.row_ptr[P] + 1] - e0) * NQ2;
    for (int it = tid; it < n_face; it += DG_THREADS) {
        asm volatile("" ::: "memory");
        const int fi = it / NQ2, q = it - fi * NQ2, code = A.bf[e0 + fi], t = code >> 2, e2 = A.neigh[code];
        const bool dir = e2 == LYMPH_BC_DIRI;
        const int Q = dir ? P : A.tet_poly[e2];
        const double* fk = &A.fk[(int64_t)t * 12];
        const double* nm = &A.ref->node_maps[(code & 3) * 16];
        const double* nt = &A.ref->nodtria2[q * 4];
        double rc[3], x[3];
#pragma unroll
        for (int r = 0; r < 3; ++r)
            rc[r] = fma(nm[r * 4], nt[0], fma(nm[r * 4 + 1], nt[1], fma(nm[r * 4 + 2], nt[2], nm[r * 4 + 3] * nt[3])));
        double L[3][PD + 1], dL[PD + 1], v[3], z[3];
#pragma unroll
        for (int d = 0; d < 3; ++d) {
            x[d] = fma(fk[d * 4], rc[0], fma(fk[d * 4 + 1], rc[1], fma(fk[d * 4 + 2], rc[2], fk[d * 4 + 3])));
            legendre_rec<PD>((x[d] - mid[d]) * ih[d], L[d], dL);
        }
        field_sf<PD>([&](int m, int j) { return s_du[j * NP + m]; }, L[0], L[1], L[2], v);
#pragma unroll
        for (int j = 0; j < 3; ++j) z[j] = v[j] = v[j] * sc;
        if (!dir) {
            double hq = 1.0, w[3];
#pragma unroll
            for (int d = 0; d < 3; ++d) {
                const double lo = A.bbox[Q * 6 + 2 * d], hi = A.bbox[Q * 6 + 2 * d + 1], i2 = 2.0 / (hi - lo);
                hq *= i2;
                legendre_rec<PD>((x[d] - 0.5 * (lo + hi)) * i2, L[d], dL);
            }
            const double *uh = A.uh + (int64_t)Q * ND, *ue = A.uex + (int64_t)Q * ND;
            field_sf<PD>([&](int m, int j) { return uh[j * NP + m] - ue[j * NP + m]; }, L[0], L[1], L[2], w);
            const double sq = sqrt(hq);
#pragma unroll
            for (int j = 0; j < 3; ++j) z[j] = fma(-sq, w[j], z[j]);
        }
        const double* n = &A.nrm[(int64_t)t * 12 + (code & 3) * 3];
        const int m = A.tet_mat[t];
        const double h = dir ? A.hk[P] : fmin(A.hk[P], A.hk[Q]);
        const double sigma = A.alpha * (double)(PD * PD) / h * (A.mat[m * 3 + 1] + 2.0 * A.mat[m * 3 + 2]);
        const double nv = n[0] * v[0] + n[1] * v[1] + n[2] * v[2], nz = n[0] * z[0] + n[1] * z[1] + n[2] * z[2];
        const double nn = n[0] * n[0] + n[1] * n[1] + n[2] * n[2], vz = v[0] * z[0] + v[1] * z[1] + v[2] * z[2];
        acc = fma(A.ref->weitria2[q] * A.area[code] * sigma, 0.5 * (nv * nz + nn * vz), acc);
    }
    // a fixed tree over the threads
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
    if ((tid & 31) == 0) s_red[tid >> 5] = acc;
    __syncthreads();
    if (tid == 0) {
        double e = 0.0;
        for (int w = 0; w < DG_THREADS / 32; ++w) e += s_red[w];
        A.partial[P] = e;
    }
}

// Deterministic sum of n values (one CTA of 1024 threads).
__global__ void __launch_bounds__(1024) k_sum(int64_t n, const double* __restrict__ v, double* out) {
    sum_fixed_order_1024(n, v, out);
}

// Sum of squares of v into *out (one CTA, fixed order).
__global__ void k_sumsq(int64_t n, const double* __restrict__ v, double* out) {
    __shared__ double red[1024];
    double s = 0.0;
    for (int64_t i = threadIdx.x; i < n; i += blockDim.x) s += v[i] * v[i];
    red[threadIdx.x] = s;
    __syncthreads();
    for (int w = blockDim.x / 2; w > 0; w >>= 1) {
        if ((int)threadIdx.x < w) red[threadIdx.x] += red[threadIdx.x + w];
        __syncthreads();
    }
    if (threadIdx.x == 0) *out = red[0];
}

// x = y / sqrt(*ss)
__global__ void k_normalize(int64_t n, const double* __restrict__ y, const double* __restrict__ ss, double* x) {
    const double inv = 1.0 / sqrt(*ss);
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
        x[i] = y[i] * inv;
}

template <int PD, typename KT, int MODE, bool INT>
int launch_step_i(lymph_ctx* c, const StepArgs& A) {
    // p = 1 in one wave of 8 to 16 CTAs per SM: an early launch unbalances the SMs and a
    // late one comes too late (48 steps of 1,728 polyhedra: 475 us in FP32, plain 390 us)
    const bool plain = PD == 1 && c->n_poly > 8 * c->sms && c->n_poly <= 16 * c->sms;
    if constexpr (MODE == MODE_STEP && PD <= 3) {
        if (c->n_poly <= c->sms && !A.abs_idx) {
            constexpr size_t bytes = SmallSmem<PD, KT>::bytes;
            LYMPH_CUDA_TRY(cudaFuncSetAttribute(k_step_small<PD, KT, INT>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                                (int)bytes));
            LYMPH_CUDA_TRY(launch_pdl(k_step_small<PD, KT, INT>, (unsigned)c->n_poly, Shape<PD>::T, c->stream, A, bytes));
            c->launches++;
            return LYMPH_OK;
        }
    }
    const auto go = [&](auto kernel) -> int {
        if (MODE == MODE_STEP && !plain) {
            LYMPH_CUDA_TRY(launch_pdl(kernel, (unsigned)c->n_poly, Shape<PD>::T, c->stream, A));
        } else {
            kernel<<<c->n_poly, Shape<PD>::T, 0, c->stream>>>(A);
            LYMPH_CUDA_TRY(cudaGetLastError());
        }
        c->launches++;
        return LYMPH_OK;
    };
    if constexpr (MODE == MODE_STEP || MODE == MODE_FIRST) {
        if (A.abs_idx) return go(k_step<PD, KT, MODE, INT, true>);
    }
    return go(k_step<PD, KT, MODE, INT, false>);
}

template <int PD, typename KT, int MODE>
int launch_step_t(lymph_ctx* c, const StepArgs& A) {
    if constexpr (PD == 2 && sizeof(KT) == 8) {
        if (A.Kex) return launch_step_i<PD, KT, MODE, true>(c, A);
    }
    return launch_step_i<PD, KT, MODE, int_columns(PD, sizeof(KT))>(c, A);
}

template <typename KT, int MODE>
int launch_step_p(lymph_ctx* c, const StepArgs& A) {
    switch (c->p) {
        case 1: return launch_step_t<1, KT, MODE>(c, A);
        case 2: return launch_step_t<2, KT, MODE>(c, A);
        case 3: return launch_step_t<3, KT, MODE>(c, A);
        case 4: return launch_step_t<4, KT, MODE>(c, A);
        default: lymph_set_error("degree not supported on the device"); return LYMPH_ERR_INVALID;
    }
}

template <int MODE>
int launch_step_mode(lymph_ctx* c, const StepArgs& A, bool fp32) {
    return fp32 ? launch_step_p<float, MODE>(c, A) : launch_step_p<double, MODE>(c, A);
}

}  // namespace

int lymph_dev_mf(lymph_ctx* c, int mode, const stepk::StepArgs& A, bool fresh);

int lymph_dev_mf_u32(lymph_ctx* c);

namespace {

// The operator pass of a step mode in the context's precision: the fused
// block-CSR kernel (FP64 or FP32 blocks) or the matrix-free neighbour kernel.
// fresh (matrix-free, MODE_STEP): the FP32 copy of u^n was left by the step before.
template <int MODE>
int launch_ctx(lymph_ctx* c, const StepArgs& A, bool fresh = false) {
    if (c->precision == LYMPH_MIXED_MF) return lymph_dev_mf(c, MODE, A, fresh);
    return launch_step_mode<MODE>(c, A, c->precision == LYMPH_MIXED);
}

StepArgs base_args(lymph_ctx* c) {
    StepArgs A;
    A.row_ptr = c->d_row_ptr; A.col = c->d_col; A.K = c->d_K; A.Kex = c->d_Kex;
    A.Minv = c->d_Minv;
    A.rhs_stat = c->d_rhs_stat; A.rhs_dyn = c->d_rhs_dyn; A.gvals = nullptr; A.step_idx = nullptr;
    A.step_off = 0; A.g = 0.0; A.u32_out = nullptr;
    A.u0 = nullptr; A.un = nullptr; A.out = nullptr; A.partial = c->d_partial; A.dt = c->dt; A.dt2 = c->dt * c->dt; A.status = c->d_status;
    A.n_poly = c->n_poly;
    A.early = trigger_early(c->p, c->n_poly, c->sms);
    A.prefetch = c->n_blocks * c->nd * c->nd * (c->precision == LYMPH_FP64 ? 8 : 4) <= STEP_PREFETCH_MAX;
    A.abs_idx = c->n_abs > 0 ? c->d_abs_idx : nullptr;
    A.Dabs = c->d_Dabs;
    A.Winv = c->d_Winv;
    return A;
}

}  // namespace

// One leapfrog step on the context stream (no rotation): reads U0/UN buffers,
// writes u^{n+1} over U0.  The caller flips c->cur afterwards.  off >= 0: step
// `off` of a run, its time-function value gvals[step_idx + off]; off < 0: the
// value g.  fresh: directly after another step of the same run.
int lymph_dev_step(lymph_ctx* c, int off, double g, bool fresh) {
    StepArgs A = base_args(c);
    A.u0 = c->d_buf[c->cur ^ 1];
    A.un = c->d_buf[c->cur];
    A.out = c->d_buf[c->cur ^ 1];
    if (off >= 0) {
        A.gvals = c->d_gvals;
        A.step_idx = c->d_step_idx;
        A.step_off = off;
    }
    A.g = g;
    return launch_ctx<MODE_STEP>(c, A, fresh);
}

// step_idx += n
int lymph_dev_bump(lymph_ctx* c, int n) {
    k_bump<<<1, 1, 0, c->stream>>>(c->d_step_idx, n);
    LYMPH_CUDA_TRY(cudaGetLastError());
    c->launches++;
    return LYMPH_OK;
}

// The FP32 copy of u^n that the first matrix-free step of a run reads.
int lymph_dev_run_start(lymph_ctx* c) { return c->precision == LYMPH_MIXED_MF ? lymph_dev_mf_u32(c) : LYMPH_OK; }

// out = M^-1 K u (u read from `u`), for the power iteration of the CFL bound.
int lymph_dev_apply(lymph_ctx* c, const double* u, double* out) {
    StepArgs A = base_args(c);
    A.un = u;
    A.u0 = u;
    A.out = out;
    return launch_ctx<MODE_APPLY>(c, A);
}

// out = K u in the context's precision (the operator apply of
// TIME_STEP_MATRIX_FREE before the mass-matrix solve).
int lymph_dev_ku(lymph_ctx* c, const double* u, double* out) {
    StepArgs A = base_args(c);
    A.un = u;
    A.u0 = u;
    A.out = out;
    return launch_ctx<MODE_KU>(c, A);
}

// out = M^-1 K u with the FP32 copy K32 of an FP64 context's blocks (the
// surrogate's predictor term, whose own error is far above FP32 rounding).
int lymph_dev_apply_fp32(lymph_ctx* c, const float* K32, const double* u, double* out) {
    StepArgs A = base_args(c);
    A.K = K32;
    A.un = u;
    A.u0 = u;
    A.out = out;
    return launch_step_p<float, MODE_APPLY>(c, A);
}

// The largest biased exponent of each FP64 block's entries (at least 200, so that
// an entry of exponent 0 is shifted out of the integer accumulator; far above
// any where the block holds infinities or NaN), a CTA per block.
__global__ void __launch_bounds__(256) k_block_exponents(const double* __restrict__ K, int nd2, int64_t block0, int32_t* ex) {
    __shared__ int s_e[8];
    const int64_t k = block0 + blockIdx.x;
    int e = 200;
    for (int i = threadIdx.x; i < nd2; i += 256) e = max(e, __double2hiint(K[k * nd2 + i]) >> 20 & 0x7ff);
    e = __reduce_max_sync(0xffffffffu, e);
    if ((threadIdx.x & 31) == 0) s_e[threadIdx.x >> 5] = e;
    __syncthreads();
    if (threadIdx.x == 0) {
        for (int w = 1; w < 8; ++w) e = max(e, s_e[w]);
        ex[k] = e == 0x7ff ? EXP_NONFINITE : e;
    }
}

// dst[i] = (float)src[i]
__global__ void k_blocks_to_f32(int64_t n, const double* __restrict__ src, float* dst) {
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
        dst[i] = (float)src[i];
}

// The FP32 copy of an FP64 context's blocks, made on first use (null when the
// context is FP32 already or the copy does not fit in device memory).
const float* lymph_dev_blocks_f32(lymph_ctx* c) {
    if (c->precision != LYMPH_FP64 || !c->have_matrices) return nullptr;
    const int64_t nK = c->n_blocks * (int64_t)c->nd * c->nd;
    if (!c->d_K32) {
        if (cudaMalloc(&c->d_K32, sizeof(float) * (size_t)nK) != cudaSuccess) {
            cudaGetLastError();  // clear the allocation failure: the caller falls back to the FP64 blocks
            c->d_K32 = nullptr;
            return nullptr;
        }
        c->device_bytes += (int64_t)sizeof(float) * nK;
        c->k32_valid = false;
    }
    if (!c->k32_valid) {
        k_blocks_to_f32<<<4096, 256, 0, c->stream>>>(nK, (const double*)c->d_K, c->d_K32);
        c->launches++;
        c->k32_valid = true;
    }
    return c->d_K32;
}

// `iters` power iterations x <- M^-1 K x / |M^-1 K x| entirely on the
// device; x must hold a nonzero start vector, y is scratch; *d_ss receives
// |M^-1 K x|^2 of the last iteration (x normalised before it).
int lymph_dev_power_iteration(lymph_ctx* c, double* x, double* y, double* d_ss, int iters) {
    const int64_t n = (int64_t)c->n_poly * c->nd;
    k_sumsq<<<1, 1024, 0, c->stream>>>(n, x, d_ss);
    k_normalize<<<1024, 256, 0, c->stream>>>(n, x, d_ss, x);
    c->launches += 2;
    for (int it = 0; it < iters; ++it) {
        LYMPH_TRY(lymph_dev_apply(c, x, y));
        k_sumsq<<<1, 1024, 0, c->stream>>>(n, y, d_ss);
        c->launches++;
        if (it + 1 < iters) {
            k_normalize<<<1024, 256, 0, c->stream>>>(n, y, d_ss, x);
            c->launches++;
        }
    }
    LYMPH_CUDA_TRY(cudaGetLastError());
    return LYMPH_OK;
}

int lymph_dev_first_step(lymph_ctx* c, double g) {
    StepArgs A = base_args(c);
    A.g = g;
    A.u0 = c->d_buf[c->cur ^ 1];
    A.un = c->d_v0;
    A.out = c->d_buf[c->cur];
    return launch_ctx<MODE_FIRST>(c, A);
}

// du . (A_dg du) per polyhedron by quadrature, then the sum.
int lymph_dev_error_dg(lymph_ctx* c, const double* uh, const double* uex, double* d_out) {
    DgArgs A;
    A.row_ptr = c->d_row_ptr; A.bf_ptr = c->d_bf_ptr; A.bf = c->d_bf; A.poly_ptr = c->d_poly_ptr;
    A.poly_tets = c->d_poly_tets; A.tet_poly = c->d_tet_poly; A.tet_mat = c->d_tet_mat; A.neigh = c->d_neigh;
    A.mat = c->d_mat; A.fk = c->d_fk; A.jdet = c->d_jdet; A.nrm = c->d_normal; A.area = c->d_area;
    A.bbox = c->d_bbox; A.hk = c->d_hk; A.ref = c->d_ref; A.uh = uh; A.uex = uex; A.alpha = c->alpha;
    A.partial = c->d_partial;
    switch (c->p) {
        case 1: k_dg_partial<1><<<c->n_poly, DG_THREADS, 0, c->stream>>>(A); break;
        case 2: k_dg_partial<2><<<c->n_poly, DG_THREADS, 0, c->stream>>>(A); break;
        case 3: k_dg_partial<3><<<c->n_poly, DG_THREADS, 0, c->stream>>>(A); break;
        case 4: k_dg_partial<4><<<c->n_poly, DG_THREADS, 0, c->stream>>>(A); break;
        default: lymph_set_error("degree not supported on the device"); return LYMPH_ERR_INVALID;
    }
    k_sum<<<1, 1024, 0, c->stream>>>(c->n_poly, c->d_partial, d_out);
    c->launches += 2;
    LYMPH_CUDA_TRY(cudaGetLastError());
    return LYMPH_OK;
}

// Leapfrog energy terms: d_out[0] = |ub - ua|^2_M (rho-weighted mass),
// d_out[1] = ub . K ua.
int lymph_dev_energy(lymph_ctx* c, const double* ua, const double* ub, double* d_out) {
    launch_l2(c, c->d_M, ub, ua);
    k_sum<<<1, 1024, 0, c->stream>>>(c->n_poly, c->d_partial, d_out);
    StepArgs A = base_args(c);
    A.u0 = ua;
    A.un = ub;
    LYMPH_TRY(launch_ctx<MODE_BILIN>(c, A));
    k_sum<<<1, 1024, 0, c->stream>>>(c->n_poly, c->d_partial, d_out + 1);
    c->launches += 3;
    LYMPH_CUDA_TRY(cudaGetLastError());
    return LYMPH_OK;
}

int lymph_dev_error_l2(lymph_ctx* c, const double* uh, const double* uex, double* d_out) {
    launch_l2(c, c->d_Mm, uh, uex);
    k_sum<<<1, 1024, 0, c->stream>>>(c->n_poly, c->d_partial, d_out);
    c->launches += 2;
    LYMPH_CUDA_TRY(cudaGetLastError());
    return LYMPH_OK;
}

// Whether the context's step kernel multiplies columns on the integer pipe: FP64
// blocks at p = 3 and 4 (48 steps, FP64 products alone -> integer columns: tetrahedra, 4
// to 5 blocks a row, p = 3, 48 / 384 / 6,000 polyhedra 0.43 / 0.93 / 10.1 -> 0.41 / 0.76 /
// 7.5 ms, p = 4 0.91 / 2.50 / 28.6 -> 0.81 / 1.76 / 20.8; 125 hexahedra 0.53 -> 0.52 and 1.22
// -> 1.08; no mesh of 21 polyhedra or more was slower), and at p = 2 on long rows (8
// blocks or more on average) from 4 CTAs per SM on: 46,861 polyhedra 45.7 -> 37.8 ms for
// 48 steps, 737 1.02 -> 0.87.  There the preparation of the coefficients cost a short row
// what it gained (hexahedra, 7 blocks: 8,000 5.64 -> 5.66 ms), a small grid more (125:
// 345 -> 405 us), and p = 1 at any size (46,767, 16 steps: 4.06 -> 4.25 ms).
bool lymph_dev_int_columns(const lymph_ctx* c) {
    if (c->precision != LYMPH_FP64) return false;
    return c->p >= 3 || (c->p == 2 && c->n_poly >= 4 * c->sms && c->n_blocks >= 8 * (int64_t)c->n_poly);
}

// The exponents of the assembled FP64 blocks that the integer columns need.
int lymph_dev_block_exponents(lymph_ctx* c) {
    if (!c->d_Kex) return LYMPH_OK;
    const int64_t chunk = 1 << 20;
    for (int64_t b0 = 0; b0 < c->n_blocks; b0 += chunk) {
        const unsigned nb = (unsigned)(c->n_blocks - b0 < chunk ? c->n_blocks - b0 : chunk);
        k_block_exponents<<<nb, 256, 0, c->stream>>>((const double*)c->d_K, c->nd * c->nd, b0, c->d_Kex);
        c->launches++;
    }
    LYMPH_CUDA_TRY(cudaGetLastError());
    return LYMPH_OK;
}
