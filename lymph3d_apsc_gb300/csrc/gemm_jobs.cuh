// gemm_jobs.cuh -- the FP32 GEMMs of the network's backward, and of its forward
// where the tensor-core kernel does not take the shapes (mpnn.cu).
//
// A training graph has a few hundred nodes, so one GEMM of the network is 15 to
// 60 MFLOP: what bounds it is how many CTAs share it and how many launches
// the step takes, not a pipe.  So
//  * a tile is 32 x 64 with 128 threads, and the four CTAs of a cluster split
//    a tile's K (for the weight gradients: the nodes), their partial sums
//    added in rank order over distributed shared memory;
//  * one launch takes two independent GEMMs (a layer's weight gradient and its
//    input gradient), one after the other in the grid;
//  * concatenations ([h a g]) are K segments (forward) or row segments (weight
//    gradient), the bias gradient is the weight gradient's row of ones, and
//    the ReLU's backward mask is applied in the epilogue that produces the
//    masked gradient.
// A training step on 424 nodes (p = 3, H = 256, L = 3) took 1.77 ms with 64 x 64
// tiles (16 CTAs for a weight gradient, looping over every node), a column sum
// per bias and a mask pass per layer (54 launches); it takes 0.45 ms (27).
#pragma once

#include <cooperative_groups.h>
#include <cuda_bf16.h>

namespace jobs {

constexpr int TM = 32, TN = 64, TK = 16, THREADS = 128, SPLIT = 4;

struct Seg {
    const float* p;
    int w, ld;   // columns, row stride
};

enum Kind {
    FWD = 0,   // C[m, n] = sum_k A[m, k] W[k, n]        A: row segments of K
    DX = 1,    // C[m, n] = sum_k A[m, k] W[n, k]        A: one segment
    DW = 2     // C[r, n] = sum_m A[m, r] dz[m, n]       A: row segments of r, then a column of ones
};
enum Epi {
    STORE = 0,      // C = v (+ bias)
    RELU = 1,       // z = v + bias, C = relu(z)
    RES_RELU = 2,   // z = v + bias, C = R + relu(z)
    GRAD = 3        // columns < n_add: C += v, with mask: dz = mask > 0 ? C : 0; the others: C2 = v
};

struct Job {
    int kind, epi, split;   // split: the cluster's CTAs share a tile's K
    int M, N, K;
    Seg a[3];
    int na;
    const __nv_bfloat16* W;   // FWD, DX
    const float* dz;          // DW
    int ldb;
    float* C;
    int ldc;
    const float *bias, *R;    // FWD
    float* z;                 // FWD: the pre-activation (may be null)
    int n_add, add;           // GRAD: columns of C, whether they accumulate (else: stored)
    const float* mask;        // GRAD (may be null)
    float *dz_out, *C2;
    int tiles_m, tiles_n;
    __host__ __device__ int ctas() const { return split ? SPLIT * tiles_m * tiles_n : (tiles_m * tiles_n + SPLIT - 1) / SPLIT * SPLIT; }
};

struct Args {
    Job j[2];
    int n;
};

__device__ __forceinline__ float seg_at(const Job& J, int row, int col) {
#pragma unroll
    for (int s = 0; s < 3; ++s) {
        if (s >= J.na) break;
        if (col < J.a[s].w) return J.a[s].p[(int64_t)row * J.a[s].ld + col];
        col -= J.a[s].w;
    }
    return 1.0f;   // DW: the column of ones
}

template <int KIND>
__device__ __forceinline__ void load(const Job& J, int m0, int n0, int k0, int k1, float (&ra)[4], float (&rb)[8]) {
    const int tid = threadIdx.x;
#pragma unroll
    for (int i = 0; i < 4; ++i) {   // A tile, [TK][TM]
        const int e = tid + i * THREADS;
        const int mm = KIND == DW ? e % TM : e / TK, kk = KIND == DW ? e / TM : e % TK;   // contiguous along the rows read
        const int m = m0 + mm, k = k0 + kk;
        ra[i] = (m < J.M && k < k1) ? (KIND == DW ? seg_at(J, k, m) : seg_at(J, m, k)) : 0.0f;
    }
#pragma unroll
    for (int i = 0; i < 8; ++i) {   // B tile, [TK][TN]
        const int e = tid + i * THREADS;
        const int nn = KIND == DX ? e / TK : e % TN, kk = KIND == DX ? e % TK : e / TN;
        const int n = n0 + nn, k = k0 + kk;
        float v = 0.0f;
        if (n < J.N && k < k1) {
            if (KIND == DW) v = J.dz[(int64_t)k * J.ldb + n];
            else v = __bfloat162float(KIND == DX ? J.W[(int64_t)n * J.ldb + k] : J.W[(int64_t)k * J.ldb + n]);
        }
        rb[i] = v;
    }
}

struct Smem {
    float A[2][TK][TM + 4];
    float B[2][TK][TN + 4];
    float red[TM][TN];
};

template <int KIND>
__device__ __forceinline__ void store(Smem& s, int b, const float (&ra)[4], const float (&rb)[8]) {
    const int tid = threadIdx.x;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const int e = tid + i * THREADS;
        if (KIND == DW) s.A[b][e / TM][e % TM] = ra[i];
        else s.A[b][e % TK][e / TK] = ra[i];
    }
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        const int e = tid + i * THREADS;
        if (KIND == DX) s.B[b][e % TK][e / TK] = rb[i];
        else s.B[b][e / TN][e % TN] = rb[i];
    }
}

// The tile's product over [k0, k1) into s.red; the next K step's operands are
// in flight in registers while this one multiplies.
template <int KIND>
__device__ __forceinline__ void tile(const Job& J, Smem& s, int m0, int n0, int k0, int k1) {
    const int tid = threadIdx.x, tx = tid % 16, ty = tid / 16;
    float acc[4][4] = {};
    float ra[4], rb[8];
    int b = 0;
    if (k0 < k1) {
        load<KIND>(J, m0, n0, k0, k1, ra, rb);
        store<KIND>(s, 0, ra, rb);
    }
    __syncthreads();
    for (int k = k0; k < k1; k += TK, b ^= 1) {
        const bool more = k + TK < k1;
        if (more) load<KIND>(J, m0, n0, k + TK, k1, ra, rb);
#pragma unroll
        for (int kk = 0; kk < TK; ++kk) {
            const float4 av = *reinterpret_cast<const float4*>(&s.A[b][kk][4 * ty]);
            const float4 bv = *reinterpret_cast<const float4*>(&s.B[b][kk][4 * tx]);
            const float a4[4] = {av.x, av.y, av.z, av.w}, b4[4] = {bv.x, bv.y, bv.z, bv.w};
#pragma unroll
            for (int r = 0; r < 4; ++r)
#pragma unroll
                for (int c = 0; c < 4; ++c) acc[r][c] = fmaf(a4[r], b4[c], acc[r][c]);
        }
        if (more) store<KIND>(s, b ^ 1, ra, rb);
        __syncthreads();
    }
#pragma unroll
    for (int r = 0; r < 4; ++r)
        *reinterpret_cast<float4*>(&s.red[4 * ty + r][4 * tx]) = make_float4(acc[r][0], acc[r][1], acc[r][2], acc[r][3]);
}

__device__ __forceinline__ void epilogue(const Job& J, int m, int n, float v) {
    if (m >= J.M || n >= J.N) return;
    if (J.epi == GRAD) {
        if (n >= J.n_add) {
            J.C2[(int64_t)m * J.ldc + n - J.n_add] = v;
            return;
        }
        const int64_t q = (int64_t)m * J.ldc + n;
        if (J.add) v += J.C[q];
        J.C[q] = v;
        if (J.mask) J.dz_out[q] = J.mask[q] > 0.0f ? v : 0.0f;
        return;
    }
    const int64_t q = (int64_t)m * J.ldc + n;
    if (J.bias) v += J.bias[n];
    if (J.epi == STORE) {
        J.C[q] = v;
        return;
    }
    if (J.z) J.z[q] = v;
    const float r = v > 0.0f ? v : 0.0f;
    J.C[q] = J.epi == RES_RELU ? J.R[q] + r : r;
}

__global__ void __cluster_dims__(SPLIT, 1, 1) __launch_bounds__(THREADS) k_gemm_jobs(const __grid_constant__ Args A) {
    namespace cg = cooperative_groups;
    __shared__ __align__(16) Smem s;
    asm volatile("griddepcontrol.wait;" ::: "memory");
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    cg::cluster_group cl = cg::this_cluster();
    const int rank = (int)cl.block_rank(), tid = threadIdx.x;
    int blk = blockIdx.x, which = 0;
    if (A.n > 1 && blk >= A.j[0].ctas()) {
        blk -= A.j[0].ctas();
        which = 1;
    }
    const Job& J = A.j[which];
    const int tile_id = J.split ? blk / SPLIT : blk;
    const bool live = tile_id < J.tiles_m * J.tiles_n;
    const int m0 = tile_id % J.tiles_m * TM, n0 = tile_id / J.tiles_m * TN;
    if (live) {
        int k0 = 0, k1 = J.K;
        if (J.split) {
            const int per = ((J.K + SPLIT - 1) / SPLIT + TK - 1) / TK * TK;
            k0 = rank * per < J.K ? rank * per : J.K;
            k1 = k0 + per < J.K ? k0 + per : J.K;
        }
        if (J.kind == FWD) tile<FWD>(J, s, m0, n0, k0, k1);
        else if (J.kind == DX) tile<DX>(J, s, m0, n0, k0, k1);
        else tile<DW>(J, s, m0, n0, k0, k1);
    }
    if (J.split) {   // the same for every CTA of the cluster
        cl.sync();
        constexpr int ROWS = TM / SPLIT;
        for (int e = tid; e < ROWS * TN; e += THREADS) {
            const int r = rank * ROWS + e / TN, c = e % TN;
            float v = 0.0f;
#pragma unroll
            for (int k = 0; k < SPLIT; ++k) v += *cl.map_shared_rank(&s.red[r][c], k);
            epilogue(J, m0 + r, n0 + c, v);
        }
        cl.sync();   // the partial sums stay until every rank has read them
    } else if (live) {
        __syncthreads();
        for (int e = tid; e < TM * TN; e += THREADS) epilogue(J, m0 + e / TN, n0 + e % TN, s.red[e / TN][e % TN]);
    }
}

// Fills in the tile counts and chooses the split: a tile's K is shared while
// the tiles alone leave SMs idle (fewer than two CTAs per SM), or, for the
// weight gradients, always (their K is the number of nodes).
inline void finish(Job& J, int sms) {
    J.tiles_m = (J.M + TM - 1) / TM;
    J.tiles_n = (J.N + TN - 1) / TN;
    J.split = J.kind == DW || J.tiles_m * J.tiles_n < 2 * sms;
}

}  // namespace jobs
