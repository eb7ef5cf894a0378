// FemPIC node-side loops and the field solve on the GPU (include/oppb_field.h).
//
// compute_node_charge_density_kernel and compute_electric_field_kernel are one thread per
// node / cell, each product and sum rounded on its own in the reference's order (this file
// is compiled with -fmad=false), so their results equal the reference's bit for bit for the
// same inputs.
//
// compute_phi of a system kept by diagonals takes the kernels of "CG on K by diagonals" below.  Any
// other system is one cooperative launch, field_newton_kernel: the grid runs init_f1_and_J, build_f1_vector and
// build_j_matrix (cell integrals added with FP64 atomics, as the reference's device
// kernels do), B = K D - F0 - F1, then Jacobi-preconditioned CG on J Y = B, D -= Y and the
// node potentials, separated by grid-wide barriers.  The iteration count is bounded by
// max_iter, every barrier is the cooperative grid's (all blocks are resident by
// construction of the launch), and no host synchronisation is needed, so a stream capture
// of the call is one graph node.  The dot products are reduced deterministically: each block
// writes its partial sum, and after the barrier every block sums all partials in block
// order, so all blocks hold the same scalars and a run repeats bit for bit.

#include <cooperative_groups.h>

#include <cstring>

#include "oppb_common.cuh"
#include "oppb_field.h"

namespace cg = cooperative_groups;

namespace oppb {
namespace {

constexpr int kFieldBlock = 256;
constexpr int kMaxCoopBlocks = 148 * 8;
constexpr int kWarps = kFieldBlock / 32;

struct FieldArgs {
    int32_t n_nodes, n_cells, neq;
    const int32_t* node_to_eq;
    const int32_t* c2n;
    const double* det_j;
    const double* n_bnd_pot;
    const int64_t* k_rowptr;
    const int32_t* k_col;
    const double* k_val;
    const double* f0;
    double* d;
    double* f1;
    const double* ion_den;
    double* potential;
    oppb_field_status* status;
    // work
    double *t1, *t2, *t3, *diag, *x, *r, *p, *q;
    double* partial_a;  // [kMaxCoopBlocks]
    double* partial_b;  // [kMaxCoopBlocks][2]
    // constants
    double n0, phi0, kte, qe, eps0, rtol, atol;
    int32_t max_iter;
    // K by diagonals (n_diag > 0): dia_val[j * neq + r] = K[r][r + dia_off[j]], offsets ascending.
    int32_t n_diag;
    int32_t dia_off[OPPB_FIELD_MAX_DIAG];
    const double* dia_val;
};

// Sum of v over the block, returned to every thread (fixed order: deterministic).
__device__ double block_sum(double v, double* sm) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(kFullMask, v, o);
    __syncthreads();  // sm may still be read by a previous call
    if (lane == 0) sm[warp] = v;
    __syncthreads();
    double s = 0.0;
#pragma unroll
    for (int w = 0; w < kWarps; w++) s += sm[w];
    return s;
}

// Sum over blocks of partial[b * stride + k], in block order, by every block.
__device__ double grid_sum(const double* partial, int stride, int k, double* sm) {
    double v = 0.0;
    for (int b = threadIdx.x; b < (int)gridDim.x; b += kFieldBlock) v += partial[b * stride + k];
    return block_sum(v, sm);
}

// Shape function a at Gauss point (i, j, k) of the 2x2x2 rule (evaluate_na in the reference's
// build_f1_vector / build_j_matrix).
__device__ __forceinline__ double shape_na(int a, int i, int j, int k) {
    const double g = __dsqrt_rn(1.0 / 3.0);
    const double li = i ? g : -g, lj = j ? g : -g, lk = k ? g : -g;
    const double ni = 0.5 * (li + 1), nj = 0.5 * (lj + 1), nk = 0.5 * (lk + 1);
    return a == 0 ? ni : a == 1 ? nj : a == 2 ? nk : ((1 - ni) - nj) - nk;
}

// init_f1_and_J (field_solver/device.cpp init_f1_kernel, init_J_kernel).
__device__ __forceinline__ void init_terms(const FieldArgs& a, int64_t tid, int64_t nth) {
    const double qe_eps0 = a.qe / a.eps0;
    for (int64_t n = tid; n < a.n_nodes; n += nth) {
        const int32_t e = a.node_to_eq[n];
        if (e >= 0) a.t1[e] = qe_eps0 * (a.ion_den[n] + a.n0 * exp((a.d[e] - a.phi0) / a.kte));
    }
    for (int64_t u = tid; u < a.neq; u += nth) {
        a.t2[u] = 0.0;
        a.t3[u] = -a.qe / a.eps0 * a.n0 * exp((a.d[u] - a.phi0) / a.kte) * (1 / a.kte);
    }
}

// build_f1_vector and build_j_matrix: per cell and unknown vertex, the 8-point integrals of
// tempNEQ1 and tempNEQ3 times the shape function, added into F1 and tempNEQ2.
__device__ __forceinline__ void add_cell_integrals(const FieldArgs& a, int64_t tid, int64_t nth) {
    for (int64_t c = tid; c < a.n_cells; c += nth) {
        const double dj = a.det_j[c];
        for (int v = 0; v < 4; v++) {
            const int32_t e = a.node_to_eq[a.c2n[c * 4 + v]];
            if (e < 0) continue;
            const double s1 = a.t1[e], s3 = a.t3[e];
            double ff1 = 0.0, ff3 = 0.0;
            for (int k = 0; k < 2; k++)
                for (int j = 0; j < 2; j++)
                    for (int i = 0; i < 2; i++) {
                        const double na = shape_na(v, i, j, k);
                        ff1 += s1 * na * dj * 1.0 * 1.0 * 1.0;
                        ff3 += s3 * na * dj * 1.0 * 1.0 * 1.0;
                    }
            atomicAdd(a.f1 + e, ff1 * (1.0 / 8.0));
            atomicAdd(a.t2 + e, ff3 * (1.0 / 8.0));
        }
    }
}

// compute_node_potential from D's values d.
__device__ __forceinline__ void node_potentials(const FieldArgs& a, const double* d, int64_t tid, int64_t nth) {
    for (int64_t n = tid; n < a.n_nodes; n += nth) {
        const int32_t e = a.node_to_eq[n];
        a.potential[n] = a.n_bnd_pot[n] + ((e >= 0) ? d[e] : 0);
    }
}

// Row u of J v (K with its diagonal replaced by du) or, with kDiag false, of K v: four column
// indices and values are loaded before their four vector gathers, so each thread keeps several
// independent loads in flight; the terms are still added one by one in column order.  K is
// read-only for the whole launch (non-coherent loads); v is not (plain loads: the vectors are
// rewritten between grid barriers).
template <bool kDiag>
__device__ __forceinline__ double row_dot(const FieldArgs& a, int64_t u, double du, const double* v) {
    if (a.n_diag > 0) {
        // By diagonals: neighbouring rows read neighbouring values of every diagonal and of v,
        // so a warp's loads are coalesced.  Offsets ascend, so the nonzero terms are added in
        // the CSR row's column order; the zeros of a diagonal where the row has no entry add
        // +0 or -0 to a sum that starts at +0 and so is never -0, which leaves it unchanged.
        double s = 0.0;
#pragma unroll 4
        for (int j = 0; j < a.n_diag; j++) {
            const int32_t off = a.dia_off[j];
            const int64_t c = u + off;
            double kv = __ldg(a.dia_val + (int64_t)j * a.neq + u);
            if (kDiag && off == 0) kv = du;
            const double vc = (c >= 0 && c < a.neq) ? v[c] : 0.0;
            s += kv * vc;
        }
        return s;
    }
    int64_t k = __ldg(a.k_rowptr + u);
    const int64_t end = __ldg(a.k_rowptr + u + 1);
    double s = 0.0;
    for (; k + 4 <= end; k += 4) {
        const int32_t c0 = __ldg(a.k_col + k), c1 = __ldg(a.k_col + k + 1);
        const int32_t c2 = __ldg(a.k_col + k + 2), c3 = __ldg(a.k_col + k + 3);
        double v0 = __ldg(a.k_val + k), v1 = __ldg(a.k_val + k + 1);
        double v2 = __ldg(a.k_val + k + 2), v3 = __ldg(a.k_val + k + 3);
        const double p0 = v[c0], p1 = v[c1], p2 = v[c2], p3 = v[c3];
        if (kDiag) {
            v0 = c0 == u ? du : v0;
            v1 = c1 == u ? du : v1;
            v2 = c2 == u ? du : v2;
            v3 = c3 == u ? du : v3;
        }
        s += v0 * p0;
        s += v1 * p1;
        s += v2 * p2;
        s += v3 * p3;
    }
    for (; k < end; k++) {
        const int32_t c = __ldg(a.k_col + k);
        const double vk = (kDiag && c == u) ? du : __ldg(a.k_val + k);
        s += vk * v[c];
    }
    return s;
}

__global__ void __launch_bounds__(kFieldBlock) field_newton_kernel(FieldArgs a) {
    cg::grid_group grid = cg::this_grid();
    __shared__ double sm[kWarps];
    const int64_t tid = (int64_t)blockIdx.x * kFieldBlock + threadIdx.x;
    const int64_t nth = (int64_t)gridDim.x * kFieldBlock;

    init_terms(a, tid, nth);
    grid.sync();

    add_cell_integrals(a, tid, nth);
    grid.sync();

    // B = K D - F0 - F1; J's diagonal = K's - tempNEQ2; CG start x = 0, r = B, p = r / diag.
    double bb = 0.0, rz = 0.0;
    for (int64_t u = tid; u < a.neq; u += nth) {
        double kd = 0.0, kuu = 0.0;
        for (int64_t k = a.k_rowptr[u]; k < a.k_rowptr[u + 1]; k++) {
            const int32_t col = a.k_col[k];
            kd += a.k_val[k] * a.d[col];
            if (col == u) kuu = a.k_val[k];
        }
        const double b = (kd - a.f0[u]) - a.f1[u];
        const double dg = kuu + (-a.t2[u]);
        a.diag[u] = dg;
        a.x[u] = 0.0;
        a.r[u] = b;
        const double z = b / dg;
        a.p[u] = z;
        bb += b * b;
        rz += b * z;
    }
    bb = block_sum(bb, sm);
    rz = block_sum(rz, sm);
    if (threadIdx.x == 0) {
        a.partial_b[blockIdx.x * 2] = bb;
        a.partial_b[blockIdx.x * 2 + 1] = rz;
    }
    grid.sync();
    bb = grid_sum(a.partial_b, 2, 0, sm);
    rz = grid_sum(a.partial_b, 2, 1, sm);
    const double b_norm = sqrt(bb);
    const double stop = fmax(a.rtol * b_norm, a.atol);
    double rr = bb;
    int it = 0;
    while (it < a.max_iter && sqrt(rr) > stop) {
        double pq = 0.0;
        for (int64_t u = tid; u < a.neq; u += nth) {  // q = J p
            const double s = row_dot<true>(a, u, a.diag[u], a.p);
            a.q[u] = s;
            pq += a.p[u] * s;
        }
        pq = block_sum(pq, sm);
        if (threadIdx.x == 0) a.partial_a[blockIdx.x] = pq;
        grid.sync();
        pq = grid_sum(a.partial_a, 1, 0, sm);
        const double alpha = rz / pq;
        double rz_new = 0.0, rr_new = 0.0;
        for (int64_t u = tid; u < a.neq; u += nth) {
            a.x[u] += alpha * a.p[u];
            const double ru = a.r[u] - alpha * a.q[u];
            a.r[u] = ru;
            rz_new += ru * (ru / a.diag[u]);
            rr_new += ru * ru;
        }
        rz_new = block_sum(rz_new, sm);
        rr_new = block_sum(rr_new, sm);
        if (threadIdx.x == 0) {
            a.partial_b[blockIdx.x * 2] = rz_new;
            a.partial_b[blockIdx.x * 2 + 1] = rr_new;
        }
        grid.sync();
        rz_new = grid_sum(a.partial_b, 2, 0, sm);
        rr_new = grid_sum(a.partial_b, 2, 1, sm);
        const double beta = rz_new / rz;
        rz = rz_new;
        rr = rr_new;
        for (int64_t u = tid; u < a.neq; u += nth) a.p[u] = a.r[u] / a.diag[u] + beta * a.p[u];
        grid.sync();
        it++;
    }

    // D -= Y (VecAXPY(D, -1, Y)), then compute_node_potential.
    for (int64_t u = tid; u < a.neq; u += nth) a.d[u] = a.d[u] - a.x[u];
    grid.sync();
    node_potentials(a, a.d, tid, nth);
    if (tid == 0) {
        a.status->iterations = it;
        a.status->converged = sqrt(rr) <= stop;
        a.status->resid = b_norm > 0.0 ? sqrt(rr) / b_norm : 0.0;
        a.status->b_norm = b_norm;
    }
}

// ------------------------------------------------------------- CG on K by diagonals
//
// The Newton step of a system stored by diagonals: two set-up kernels over the whole chip, one
// persistent CG kernel, one kernel that takes the step and writes the node potentials.
//
// What bounds the CG is neither DRAM nor arithmetic but what an iteration does one after the
// other: grid barriers, passes over vectors in memory and the loads of K.  So each block owns a
// contiguous range of rows and keeps x, r, z and the diagonal of its rows in registers, as many
// diagonals of K as fit in shared memory (the others are streamed from L2), and the search
// direction p of its rows and of the rows its diagonals reach in a shared-memory window.  Only
// z = r / diag crosses blocks: every block forms p = z + beta p on its whole window itself (the
// same operations on the same values in every block), which saves the third barrier.  An
// iteration is: window update, product and p.q, reduction A, x, r and z, r.z and r.r, reduction B.
//
// Systems of up to kClusterNeq unknowns run as one thread-block cluster, whose barrier and
// distributed shared memory replace the polled slots in global memory.  kCluster = false is a
// cooperative launch of one block per SM.  At 458,591 unknowns (15 diagonals) an iteration takes
// 13.4 us instead of 25.9 in field_newton_kernel, at 138,303 8.0 instead of 14.5.  Of the 13.4 the
// product takes 5 (K streamed from L2, then shared memory), the two reductions 6.

constexpr int kCgMaxThreads = 640;  // 102 registers a thread
constexpr int kCgMaxRows = 8;       // rows a thread
constexpr int kCgMinRows = 64;      // rows a block, where there are as many
constexpr int kStage = 4;           // window loads in flight a thread
constexpr int kCgMaxCluster = 16;
constexpr int kCgMaxWarps = kCgMaxThreads / 32;
constexpr int kCgMaxBlocks = 160;  // of the grid form

// One block's sums in global memory: each value and the number of the reduction it belongs to are
// one 16-byte word, so that a block that reads the number has the value too.  A slot fills a
// 128-byte line: every block polls every slot, and packed slots would all be served by a few L2
// slices.
struct __align__(16) CgWord {
    double value;
    unsigned long long turn;
};
struct __align__(128) CgSlot {
    CgWord value[2];
    CgWord unused[6];
};

__device__ __forceinline__ void post_word(CgWord* p, double v, unsigned long long turn) {
    const unsigned __int128 w = ((unsigned __int128)turn << 64) | (unsigned long long)__double_as_longlong(v);
    asm volatile("st.relaxed.gpu.global.b128 [%0], %1;" ::"l"(p), "q"(w) : "memory");
}
__device__ __forceinline__ bool poll_word(const CgWord* p, unsigned long long turn, double& v) {
    unsigned __int128 w;
    asm volatile("ld.relaxed.gpu.global.b128 %0, [%1];" : "=q"(w) : "l"(p) : "memory");
    v = __longlong_as_double((long long)(unsigned long long)w);
    return (unsigned long long)(w >> 64) == turn;
}

// Reduction scratch of a block, indexed [value].
struct CgShared {
    double part[2][2][kCgMaxCluster * kCgMaxWarps];  // cluster form: the sums of every warp of the cluster
    double warp[2][kCgMaxWarps];                     // grid form: the block's warps
    double sum[2];
    int failed;
};

struct CgArgs {
    FieldArgs f;
    int32_t rows;      // rows a block owns
    int32_t lo, hi;    // the window reaches lo rows before and hi rows after them
    int32_t smem_diag; // the last smem_diag diagonals are kept in shared memory
    int32_t max_polls; // bound of a wait of the grid form
    CgSlot* slots;     // [2][gridDim.x], grid form; zeroed before the launch
    int* gave_up;      // 1 once a block's wait has run out; zeroed before the launch
    double* next_d;    // [neq] D - Y
};

// Sums over the lanes that hold one value: all 32 for kValues = 1, else lanes 0..15 hold the first
// and 16..31 the second.
template <int kValues>
__device__ __forceinline__ double lane_sum(double v) {
#pragma unroll
    for (int o = kValues == 2 ? 8 : 16; o > 0; o >>= 1) v += __shfl_xor_sync(kFullMask, v, o);
    return v;
}

// Sum of v (its first kValues doubles) over all threads of all blocks, the same bits in every
// thread.  With kBarrier it is also a barrier of all blocks: what any thread wrote before, every
// thread sees after.  turn counts the reductions of the launch from 1.
//
// Two values travel as one: half the lanes reduce the first, half the second, which shortens the
// chain of shuffles.  Cluster form: every warp stores its sums into every block's shared memory,
// then one cluster barrier.  Grid form: the block's sums go to its slot together with the turn, and
// warp 0 polls the slots of all blocks, so that the reduction and the barrier are one round trip
// through L2 (a cooperative-groups grid barrier with the partial sums beside it took 7 us).  The
// blocks are all resident (cooperative launch); a wait that runs out sets sh.failed, on which the block
// ends, and *gave_up, on which field_finish_kernel drops the step of all blocks.
template <int kValues, bool kBarrier, bool kCluster>
__device__ __forceinline__ double2 cg_all_sum(double2 in, CgShared& sh, const CgArgs& c, unsigned turn) {
    constexpr int kLanes = 32 / kValues;  // lanes a value
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, n_warps = blockDim.x >> 5;
    const int sub = lane % kLanes, value = lane / kLanes;
    const int n_blocks = (int)gridDim.x;
    double v = in.x;
    if (kValues == 2) {
        const double other = __shfl_xor_sync(kFullMask, value == 0 ? in.y : in.x, 16);
        v = (value == 0 ? in.x : in.y) + other;
    }
    v = lane_sum<kValues>(v);
    if (kCluster) {
        double* mine = &sh.part[turn & 1][value][blockIdx.x * n_warps + warp];
        if (sub < n_blocks) *cg::this_cluster().map_shared_rank(mine, sub) = v;
        cg::this_cluster().sync();
        double2 s = make_double2(0.0, 0.0);
        for (int w = lane; w < n_blocks * n_warps; w += 32) {
            s.x += sh.part[turn & 1][0][w];
            if (kValues == 2) s.y += sh.part[turn & 1][1][w];
        }
        v = s.x;
        if (kValues == 2) {
            const double other = __shfl_xor_sync(kFullMask, value == 0 ? s.y : s.x, 16);
            v = (value == 0 ? s.x : s.y) + other;
        }
        v = lane_sum<kValues>(v);
        if (kValues == 1) return make_double2(v, 0.0);
        return make_double2(__shfl_sync(kFullMask, v, 0), __shfl_sync(kFullMask, v, 16));
    }
    if (sub == 0) sh.warp[value][warp] = v;
    __syncthreads();
    if (warp == 0) {
        v = 0.0;
        for (int w = sub; w < n_warps; w += kLanes) v += sh.warp[value][w];
        v = lane_sum<kValues>(v);
        CgSlot* at = c.slots + (turn & 1) * n_blocks;
        if (sub == 0) {
            if (kBarrier) __threadfence();
            post_word(&at[blockIdx.x].value[value], v, turn);
        }
        constexpr int kSlots = (kCgMaxBlocks + kLanes - 1) / kLanes;
        double x[kSlots] = {};
        bool all = false;
        for (int poll = 0; !all && poll < c.max_polls; poll++) {
            bool here = true;
#pragma unroll
            for (int k = 0; k < kSlots; k++) {
                const int b = sub + kLanes * k;
                x[k] = 0.0;
                if (b < n_blocks) {
                    const bool posted = poll_word(&at[b].value[value], turn, x[k]);
                    here = here && posted;
                }
            }
            all = __all_sync(kFullMask, here);
        }
        if (kBarrier) __threadfence();
        v = 0.0;
#pragma unroll
        for (int k = 0; k < kSlots; k++) v += x[k];
        v = lane_sum<kValues>(v);
        if (sub == 0) sh.sum[value] = v;
        if (lane == 0 && !all) sh.failed = *c.gave_up = 1;
    }
    __syncthreads();
    return make_double2(sh.sum[0], kValues == 2 ? sh.sum[1] : 0.0);
}

template <int kRows, bool kCluster>
__global__ void __launch_bounds__(kCgMaxThreads, 1) field_cg_kernel(const __grid_constant__ CgArgs c) {
    extern __shared__ double dyn[];
    __shared__ CgShared sh;
    const FieldArgs& a = c.f;
    const int32_t r0 = (int32_t)blockIdx.x * c.rows;
    const int32_t n_own = max(0, min(c.rows, a.neq - r0));
    const int32_t width = c.rows + c.lo + c.hi;
    double* pw = dyn;          // p of rows [r0 - lo, r0 + rows + hi)
    double* km = dyn + width;  // [smem_diag][rows]
    double* zg = a.q;          // z of all rows, the only vector blocks exchange
    unsigned turn = 1;
    // A block's shared memory may be written by the others only once it runs, which being scheduled
    // together does not say: all have started before the first reduction stores into all.
    if (kCluster) cg::this_cluster().sync();
    if (threadIdx.x == 0) sh.failed = 0;
    for (int32_t i = threadIdx.x; i < width; i += blockDim.x) pw[i] = 0.0;
    const int32_t stream_diag = a.n_diag - c.smem_diag;
    for (int32_t j = 0; j < c.smem_diag; j++)
        for (int32_t i = threadIdx.x; i < n_own; i += blockDim.x)
            km[(int64_t)j * c.rows + i] = __ldg(a.dia_val + (int64_t)(stream_diag + j) * a.neq + r0 + i);

    // B = K D - F0 - F1, J's diagonal, z = r / diag (p starts as z).
    double x[kRows], r[kRows], dg[kRows], z[kRows];
    double2 v = make_double2(0.0, 0.0);
#pragma unroll
    for (int k = 0; k < kRows; k++) {
        const int32_t i = threadIdx.x + k * blockDim.x;
        x[k] = 0.0, r[k] = 0.0, dg[k] = 1.0, z[k] = 0.0;
        if (i >= n_own) continue;
        const int64_t u = r0 + i;
        double kd = 0.0, kuu = 0.0;
        for (int64_t e = __ldg(a.k_rowptr + u); e < __ldg(a.k_rowptr + u + 1); e++) {
            const int32_t col = __ldg(a.k_col + e);
            const double kv = __ldg(a.k_val + e);
            kd += kv * a.d[col];
            if (col == u) kuu = kv;
        }
        r[k] = (kd - a.f0[u]) - a.f1[u];
        dg[k] = kuu + (-a.t2[u]);
        z[k] = r[k] / dg[k];
        __stcg(zg + u, z[k]);
        v.x += r[k] * z[k];
        v.y += r[k] * r[k];
    }
    v = cg_all_sum<2, true, kCluster>(v, sh, c, turn++);
    double rz = v.x, rr = v.y;
    const double b_norm = sqrt(rr);
    const double stop = fmax(a.rtol * b_norm, a.atol);
    double beta = 0.0;
    int it = 0;
    bool failed = !kCluster && sh.failed;
    while (!failed && it < a.max_iter && sqrt(rr) > stop) {
        // p = z + beta p over the window: the block's own rows from registers, the rest with kStage
        // loads of z in flight a thread.
        const int32_t halo = c.lo + c.hi;
        for (int32_t i0 = threadIdx.x; i0 < halo; i0 += kStage * blockDim.x) {
            double zw[kStage];
#pragma unroll
            for (int k = 0; k < kStage; k++) {
                int32_t i = i0 + k * blockDim.x;
                const bool in = i < halo;
                if (i >= c.lo) i += c.rows;
                const int32_t u = r0 - c.lo + i;
                zw[k] = in && (uint32_t)u < (uint32_t)a.neq ? __ldcg(zg + u) : 0.0;
            }
#pragma unroll
            for (int k = 0; k < kStage; k++) {
                int32_t i = i0 + k * blockDim.x;
                const bool in = i < halo;
                if (i >= c.lo) i += c.rows;
                if (in) pw[i] = zw[k] + beta * pw[i];
            }
        }
#pragma unroll
        for (int k = 0; k < kRows; k++) {
            const int32_t i = threadIdx.x + k * blockDim.x;
            if (i < n_own) pw[c.lo + i] = z[k] + beta * pw[c.lo + i];
        }
        __syncthreads();
        // The product, the diagonals in ascending order of their offset: each row's terms in
        // column order.  Threads past the block's rows repeat its last one and drop the result.
        double s[kRows];
        int32_t row[kRows];
#pragma unroll
        for (int k = 0; k < kRows; k++) {
            s[k] = 0.0;
            row[k] = min((int32_t)(threadIdx.x + k * blockDim.x), n_own - 1);
        }
#pragma unroll 4
        for (int32_t j = 0; j < stream_diag; j++) {
            const int32_t off = a.dia_off[j];
            const double* kj = a.dia_val + (int64_t)j * a.neq + r0;
            const double* pj = pw + c.lo + off;
#pragma unroll
            for (int k = 0; k < kRows; k++) {
                double kv = __ldg(kj + row[k]);
                kv = off == 0 ? dg[k] : kv;
                s[k] += kv * pj[row[k]];
            }
        }
#pragma unroll 3
        for (int32_t j = stream_diag; j < a.n_diag; j++) {
            const int32_t off = a.dia_off[j];
            const double* kj = km + (j - stream_diag) * c.rows;
            const double* pj = pw + c.lo + off;
#pragma unroll
            for (int k = 0; k < kRows; k++) {
                double kv = kj[row[k]];
                kv = off == 0 ? dg[k] : kv;
                s[k] += kv * pj[row[k]];
            }
        }
        v = make_double2(0.0, 0.0);
#pragma unroll
        for (int k = 0; k < kRows; k++) {
            const int32_t i = threadIdx.x + k * blockDim.x;
            if (i < n_own) v.x += pw[i + c.lo] * s[k];
        }
        v = cg_all_sum<1, false, kCluster>(v, sh, c, turn++);
        failed = !kCluster && sh.failed;
        if (failed) break;
        const double alpha = rz / v.x;
        v = make_double2(0.0, 0.0);
#pragma unroll
        for (int k = 0; k < kRows; k++) {
            const int32_t i = threadIdx.x + k * blockDim.x;
            if (i >= n_own) continue;
            x[k] += alpha * pw[i + c.lo];
            r[k] = r[k] - alpha * s[k];
            z[k] = r[k] / dg[k];
            __stcg(zg + r0 + i, z[k]);
            v.x += r[k] * z[k];
            v.y += r[k] * r[k];
        }
        v = cg_all_sum<2, true, kCluster>(v, sh, c, turn++);
        failed = !kCluster && sh.failed;
        if (failed) break;
        beta = v.x / rz;
        rz = v.x;
        rr = v.y;
        it++;
    }
    // D - Y (VecAXPY(D, -1, Y)), which field_finish_kernel makes D.
#pragma unroll
    for (int k = 0; k < kRows; k++) {
        const int32_t i = threadIdx.x + k * blockDim.x;
        if (i < n_own) c.next_d[r0 + i] = a.d[r0 + i] - x[k];
    }
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        a.status->iterations = it;
        a.status->converged = sqrt(rr) <= stop;
        a.status->resid = b_norm > 0.0 ? sqrt(rr) / b_norm : 0.0;
        a.status->b_norm = b_norm;
    }
}

__global__ void __launch_bounds__(kFieldBlock) field_init_kernel(const __grid_constant__ FieldArgs a,
                                                                  CgSlot* slots, int n_slots, int* gave_up) {
    if ((int)(blockIdx.x * kFieldBlock + threadIdx.x) < n_slots)
        slots[blockIdx.x * kFieldBlock + threadIdx.x] = CgSlot{};
    if (blockIdx.x == 0 && threadIdx.x == 0) *gave_up = 0;
    init_terms(a, (int64_t)blockIdx.x * kFieldBlock + threadIdx.x, (int64_t)gridDim.x * kFieldBlock);
}

__global__ void __launch_bounds__(kFieldBlock) field_cells_kernel(const __grid_constant__ FieldArgs a) {
    add_cell_integrals(a, (int64_t)blockIdx.x * kFieldBlock + threadIdx.x, (int64_t)gridDim.x * kFieldBlock);
}

// D and the node potentials of the step, unless a block of field_cg_kernel gave up: then D stays as it
// was, whichever blocks ended their CG, and the status says not converged.
__global__ void __launch_bounds__(kFieldBlock) field_finish_kernel(const __grid_constant__ FieldArgs a, const int* gave_up,
                                                                    const double* next_d) {
    const int64_t tid = (int64_t)blockIdx.x * kFieldBlock + threadIdx.x, nth = (int64_t)gridDim.x * kFieldBlock;
    const bool failed = *gave_up != 0;
    node_potentials(a, failed ? a.d : next_d, tid, nth);
    if (!failed)
        for (int64_t u = tid; u < a.neq; u += nth) a.d[u] = next_d[u];
    else if (tid == 0)
        a.status->converged = 0;
}

__global__ void __launch_bounds__(256) node_charge_density_kernel(double* den, const double* vol, double spwt,
                                                                   int32_t n) {
    const int64_t i = (int64_t)blockIdx.x * 256 + threadIdx.x;
    if (i < n) den[i] *= (spwt / vol[i]);
}

__global__ void __launch_bounds__(256) electric_field_kernel(const int32_t* c2n, oppb_cell_layout nl,
                                                             const double* sd, oppb_cell_layout sl,
                                                             const double* phi, double* ef, oppb_cell_layout el,
                                                             int32_t n, int32_t accumulate) {
    const int64_t c = (int64_t)blockIdx.x * 256 + threadIdx.x;
    if (c >= n) return;
    double p[4];
#pragma unroll
    for (int v = 0; v < 4; v++) p[v] = __ldg(phi + __ldg(c2n + c * nl.cell_stride + v * nl.comp_stride));
    const double* s = sd + c * sl.cell_stride;
#pragma unroll
    for (int dim = 0; dim < 3; dim++) {
        const double c1 = __ldg(s + (0 * 3 + dim) * sl.comp_stride) * p[0];
        const double c2 = __ldg(s + (1 * 3 + dim) * sl.comp_stride) * p[1];
        const double c3 = __ldg(s + (2 * 3 + dim) * sl.comp_stride) * p[2];
        const double c4 = __ldg(s + (3 * 3 + dim) * sl.comp_stride) * p[3];
        double* e = ef + c * el.cell_stride + dim * el.comp_stride;
        *e = (accumulate ? *e : 0.0) - (c1 + c2 + c3 + c4);
    }
}

// Doubles mapped to 64-bit words whose unsigned order is the doubles' order (negative values
// complemented, positive ones with the sign bit set), so atomicMax on the words is a max.
__device__ __forceinline__ unsigned long long order_key(double v) {
    const unsigned long long b = (unsigned long long)__double_as_longlong(v);
    return (b >> 63) ? ~b : (b | 0x8000000000000000ull);
}
__device__ unsigned long long g_max_key;

__global__ void __launch_bounds__(256) reduce_max_kernel(const double* x, int64_t n, int32_t absolute) {
    __shared__ unsigned long long sm[8];
    unsigned long long k = 0ull;  // below every key of a non-NaN double
    for (int64_t i = (int64_t)blockIdx.x * 256 + threadIdx.x; i < n; i += (int64_t)gridDim.x * 256) {
        const double v = absolute ? fabs(x[i]) : x[i];
        const unsigned long long kv = order_key(v);
        k = kv > k ? kv : k;
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        const unsigned long long other = __shfl_xor_sync(kFullMask, k, o);
        k = other > k ? other : k;
    }
    if ((threadIdx.x & 31) == 0) sm[threadIdx.x >> 5] = k;
    __syncthreads();
    if (threadIdx.x == 0) {
        for (int w = 1; w < 8; w++) k = sm[w] > k ? sm[w] : k;
        atomicMax(&g_max_key, k);
    }
}

// How the CG on K by diagonals is launched.
struct CgPlan {
    int rows = 0;       // rows a block; 0 = the system does not fit this kernel
    int blocks = 0;
    int threads = 0;
    int rows_thread = 0;
    int smem_diag = 0;
    size_t smem = 0;
    int smem_max = 0;   // what the device gives a block
    bool cluster = false;
};

// Up to this many unknowns the CG runs as one cluster, above as one block per SM.  Microseconds an
// iteration, cluster / grid: 4.3 / 6.1 at 4,719 unknowns, 6.1 / 6.4 at 18,207, 9.0 / 6.3 at 34,839
// (all in field_newton_kernel: 12.9, 13.7, 13.4).
constexpr int kClusterNeq = 18432;
static_assert(kClusterNeq <= kCgMaxCluster * kCgMaxThreads * 2, "a cluster's threads have one or two rows");

CgPlan cg_plan(int32_t neq, int32_t n_diag, int32_t lo, int32_t hi, int sms, int smem_max, bool cluster) {
    CgPlan p;
    p.cluster = cluster;
    p.smem_max = smem_max;
    const int most = cluster ? kCgMaxCluster : sms < kCgMaxBlocks ? sms : kCgMaxBlocks;
    p.rows = ceil_div(neq, most);
    if (p.rows < kCgMinRows) p.rows = kCgMinRows;
    p.blocks = ceil_div(neq, p.rows);
    p.rows_thread = ceil_div(p.rows, kCgMaxThreads);
    const int64_t window = ((int64_t)p.rows + lo + hi) * (int64_t)sizeof(double);
    if (p.rows_thread > kCgMaxRows || window > smem_max) return CgPlan{};
    p.threads = (ceil_div(p.rows, p.rows_thread) + 31) / 32 * 32;
    p.smem_diag = (int)((smem_max - window) / ((int64_t)p.rows * (int64_t)sizeof(double)));
    if (p.smem_diag > n_diag) p.smem_diag = n_diag;
    p.smem = (size_t)(window + (int64_t)p.smem_diag * p.rows * (int64_t)sizeof(double));
    return p;
}

// field_cg_kernel's launch by a plan: its attributes set and its configuration filled in.
struct CgLaunch {
    cudaLaunchConfig_t cfg{};
    cudaLaunchAttribute attr{};
};
template <int kRows, bool kCluster>
int prepare_cg(const CgPlan& p, CgLaunch& l, cudaStream_t s) {
    auto kernel = field_cg_kernel<kRows, kCluster>;
    // The attribute is the kernel's, for all threads and graphs: always the device's most, so that the
    // solve of a smaller system cannot take it back between another's call here and its launch.
    if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, p.smem_max) != cudaSuccess)
        return OPPB_ERR_LAUNCH;
    if (kCluster && p.blocks > 8 &&
        cudaFuncSetAttribute(kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) != cudaSuccess)
        return OPPB_ERR_LAUNCH;
    l.cfg.gridDim = dim3(p.blocks);
    l.cfg.blockDim = dim3(p.threads);
    l.cfg.dynamicSmemBytes = p.smem;
    l.cfg.stream = s;
    if (kCluster) {
        l.attr.id = cudaLaunchAttributeClusterDimension;
        l.attr.val.clusterDim.x = (unsigned)p.blocks;
        l.attr.val.clusterDim.y = l.attr.val.clusterDim.z = 1;
    } else {
        l.attr.id = cudaLaunchAttributeCooperative;
        l.attr.val.cooperative = 1;
    }
    l.cfg.attrs = &l.attr;
    l.cfg.numAttrs = 1;
    return OPPB_OK;
}

template <int kRows, bool kCluster>
int launch_cg(const CgPlan& p, CgArgs& c, cudaStream_t s) {
    CgLaunch l;
    const int rc = prepare_cg<kRows, kCluster>(p, l, s);
    if (rc) return rc;
    return cudaLaunchKernelEx(&l.cfg, field_cg_kernel<kRows, kCluster>, c) == cudaSuccess ? OPPB_OK : OPPB_ERR_LAUNCH;
}

// Whether the device can place the plan's cluster: 16 blocks with most of an SM's shared memory each need
// as many SMs of one GPC, which a partition of the GPU may not have.
template <int kRows>
bool cluster_fits(const CgPlan& p) {
    CgLaunch l;
    int clusters = 0;
    if (prepare_cg<kRows, true>(p, l, nullptr) == OPPB_OK &&
        cudaOccupancyMaxActiveClusters(&clusters, field_cg_kernel<kRows, true>, &l.cfg) == cudaSuccess && clusters > 0)
        return true;
    cudaGetLastError();  // the answer is no, not an error of this call
    return false;
}

int launch_cg_rows(const CgPlan& p, CgArgs& c, cudaStream_t s) {
    if (p.cluster) return p.rows_thread == 1 ? launch_cg<1, true>(p, c, s) : launch_cg<2, true>(p, c, s);
    switch (p.rows_thread) {
        case 1: return launch_cg<1, false>(p, c, s);
        case 2: return launch_cg<2, false>(p, c, s);
        case 3: return launch_cg<3, false>(p, c, s);
        case 4: return launch_cg<4, false>(p, c, s);
        case 5: return launch_cg<5, false>(p, c, s);
        case 6: return launch_cg<6, false>(p, c, s);
        case 7: return launch_cg<7, false>(p, c, s);
        default: return launch_cg<8, false>(p, c, s);
    }
}

// The plan for this system on the current device; rows = 0 when it takes field_newton_kernel.  A system
// whose cluster cannot be placed takes the grid form, from kCgMinRows unknowns on (below, the slots
// would not fit in its work space).
int make_cg_plan(const FieldArgs& a, bool no_cluster, CgPlan* plan, int32_t* lo, int32_t* hi) {
    *plan = CgPlan{};
    if (a.n_diag <= 0 || a.neq <= 0) return OPPB_OK;
    int64_t first = 0, last = 0;
    for (int j = 0; j < a.n_diag; j++) {
        first = a.dia_off[j] < first ? a.dia_off[j] : first;
        last = a.dia_off[j] > last ? a.dia_off[j] : last;
        if (j > 0 && a.dia_off[j] <= a.dia_off[j - 1]) return OPPB_OK;
    }
    if (-first >= a.neq || last >= a.neq) return OPPB_OK;
    *lo = (int32_t)-first, *hi = (int32_t)last;
    int dev = 0, sms = 0, coop = 0, smem = 0;
    if (cudaGetDevice(&dev) != cudaSuccess ||
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess ||
        cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, dev) != cudaSuccess ||
        cudaDeviceGetAttribute(&smem, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev) != cudaSuccess)
        return OPPB_ERR_LAUNCH;
    smem -= (int)sizeof(CgShared) + 64;  // the kernel's static part
    if (a.neq <= kClusterNeq && !no_cluster) {
        *plan = cg_plan(a.neq, a.n_diag, *lo, *hi, sms, smem, true);
        if (plan->rows && !(plan->rows_thread == 1 ? cluster_fits<1>(*plan) : cluster_fits<2>(*plan))) *plan = CgPlan{};
    }
    if (!plan->rows && coop && a.neq >= kCgMinRows) *plan = cg_plan(a.neq, a.n_diag, *lo, *hi, sms, smem, false);
    return OPPB_OK;
}

int solve_by_diagonals(const FieldArgs& a, const CgPlan& p, int32_t lo, int32_t hi, int32_t max_polls, cudaStream_t s) {
    const int most = 148 * 8;
    const int eq_grid = ceil_div(a.n_nodes, kFieldBlock), cell_grid = ceil_div(a.n_cells, kFieldBlock);
    CgArgs c{};
    c.f = a;
    c.rows = p.rows, c.lo = lo, c.hi = hi, c.smem_diag = p.smem_diag, c.max_polls = max_polls;
    c.next_d = a.diag;  // of the work space too: this path keeps the diagonal in registers
    c.gave_up = reinterpret_cast<int*>(a.partial_a);
    // The slots lie in the vectors x, r and p of the work space, which this path keeps on chip:
    // 32 doubles a block of kCgMinRows rows or more, a last one with fewer, and the alignment.
    static_assert(3 * kCgMinRows >= 2 * 32 + 16, "the slots fit");
    c.slots = reinterpret_cast<CgSlot*>((reinterpret_cast<uintptr_t>(a.x) + 127) & ~(uintptr_t)127);
    const int n_slots = p.cluster ? 0 : 2 * p.blocks;
    const int slot_grid = ceil_div(n_slots, kFieldBlock);
    const int init_grid = eq_grid < most ? (eq_grid > slot_grid ? eq_grid : slot_grid) : most;
    field_init_kernel<<<init_grid, kFieldBlock, 0, s>>>(a, c.slots, n_slots, c.gave_up);
    field_cells_kernel<<<cell_grid, kFieldBlock, 0, s>>>(a);
    const int rc = launch_cg_rows(p, c, s);
    if (rc) return rc;
    field_finish_kernel<<<eq_grid < most ? eq_grid : most, kFieldBlock, 0, s>>>(a, c.gave_up, c.next_d);
    count_launches(4);
    return launch_status();
}

int coop_grid(int* blocks) {
    int dev = 0, sms = 0, per_sm = 0, coop = 0;
    if (cudaGetDevice(&dev) != cudaSuccess ||
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess ||
        cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, dev) != cudaSuccess ||
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, field_newton_kernel, kFieldBlock, 0) != cudaSuccess)
        return OPPB_ERR_LAUNCH;
    if (!coop || per_sm <= 0) return OPPB_ERR_LAUNCH;
    const int want = sms * (per_sm < 4 ? per_sm : 4);
    *blocks = want < kMaxCoopBlocks ? want : kMaxCoopBlocks;
    return OPPB_OK;
}

}  // namespace
}  // namespace oppb

extern "C" size_t oppb_field_work_doubles(int32_t neq) {
    if (neq < 0) return 0;
    return 8 * (size_t)(neq > 0 ? neq : 1) + 3 * (size_t)oppb::kMaxCoopBlocks;
}

extern "C" int oppb_node_charge_density(double* n_charge_den, const double* n_vol, double spwt, int32_t n_nodes,
                                        void* stream) {
    if (n_nodes < 0 || (n_nodes > 0 && (!n_charge_den || !n_vol))) return OPPB_ERR_ARG;
    if (n_nodes == 0) return OPPB_OK;
    oppb::node_charge_density_kernel<<<oppb::ceil_div(n_nodes, 256), 256, 0, oppb::as_stream(stream)>>>(
        n_charge_den, n_vol, spwt, n_nodes);
    oppb::count_launches(1);
    return oppb::launch_status();
}

extern "C" int oppb_electric_field_ex(const int32_t* c2n, oppb_cell_layout c2n_layout, const double* c_sd,
                                      oppb_cell_layout sd_layout, const double* node_potential, double* c_ef,
                                      oppb_cell_layout ef_layout, int32_t n_cells, int32_t accumulate,
                                      void* stream) {
    if (n_cells < 0 || (accumulate != 0 && accumulate != 1)) return OPPB_ERR_ARG;
    if (n_cells == 0) return OPPB_OK;
    if (!c2n || !c_sd || !node_potential || !c_ef) return OPPB_ERR_ARG;
    oppb::electric_field_kernel<<<oppb::ceil_div(n_cells, 256), 256, 0, oppb::as_stream(stream)>>>(
        c2n, c2n_layout, c_sd, sd_layout, node_potential, c_ef, ef_layout, n_cells, accumulate);
    oppb::count_launches(1);
    return oppb::launch_status();
}

extern "C" int oppb_electric_field(const int32_t* c2n, const double* c_sd, const double* node_potential,
                                   double* c_ef, int32_t ef_stride, int32_t n_cells, void* stream) {
    if (ef_stride < 3) return OPPB_ERR_ARG;
    return oppb_electric_field_ex(c2n, oppb_cell_layout{4, 1}, c_sd, oppb_cell_layout{12, 1}, node_potential, c_ef,
                                  oppb_cell_layout{ef_stride, 1}, n_cells, 0, stream);
}

extern "C" int oppb_reduce_max(const double* x, int64_t n, int32_t absolute, double init, double* result,
                               void* stream) {
    if (!result || n < 0 || (n > 0 && !x) || (absolute != 0 && absolute != 1)) return OPPB_ERR_ARG;
    *result = init;
    if (n == 0) return OPPB_OK;
    cudaStream_t s = oppb::as_stream(stream);
    unsigned long long* key = nullptr;
    if (cudaGetSymbolAddress(reinterpret_cast<void**>(&key), oppb::g_max_key) != cudaSuccess ||
        cudaMemsetAsync(key, 0, sizeof(unsigned long long), s) != cudaSuccess)
        return OPPB_ERR_LAUNCH;
    const int blocks = oppb::ceil_div(n, 256) < 148 * 8 ? oppb::ceil_div(n, 256) : 148 * 8;
    oppb::reduce_max_kernel<<<blocks, 256, 0, s>>>(x, n, absolute);
    oppb::count_launches(1);
    unsigned long long k = 0;
    if (cudaMemcpyAsync(&k, key, sizeof k, cudaMemcpyDeviceToHost, s) != cudaSuccess ||
        cudaStreamSynchronize(s) != cudaSuccess)
        return OPPB_ERR_LAUNCH;
    if (k != 0ull) {  // decode the largest key (0 = no value, n > 0 makes that impossible)
        const unsigned long long b = (k >> 63) ? (k & 0x7fffffffffffffffull) : ~k;
        double v;
        memcpy(&v, &b, sizeof v);
        if (v > *result) *result = v;  // MAX(value, init) of the reference's kernels
    }
    return oppb::launch_status();
}

extern "C" int oppb_field_solve_ex(const oppb_field_device* f, const oppb_field_consts* c, const double* ion_den,
                                   double* node_potential, oppb_field_status* status, const oppb_field_options* options,
                                   void* stream) {
    using namespace oppb;
    if (!f || !c || !ion_den || !node_potential || !status || !options || options->max_polls < 0) return OPPB_ERR_ARG;
    if (f->n_nodes <= 0 || f->n_cells <= 0 || f->neq < 0 || !f->node_to_eq || !f->c2n || !f->det_j ||
        !f->n_bnd_pot || !f->k_rowptr || !f->d || !f->f1 || !f->work || !f->f0 || (f->neq > 0 && (!f->k_col ||
        !f->k_val)))
        return OPPB_ERR_ARG;
    if (c->max_iter < 0 || !(c->kte != 0.0) || !(c->eps0 != 0.0) || !(c->rtol >= 0.0) || !(c->atol >= 0.0))
        return OPPB_ERR_ARG;
    const size_t n = (size_t)(f->neq > 0 ? f->neq : 1);
    double* w = f->work;
    FieldArgs a{};
    a.n_nodes = f->n_nodes, a.n_cells = f->n_cells, a.neq = f->neq;
    a.node_to_eq = f->node_to_eq, a.c2n = f->c2n, a.det_j = f->det_j, a.n_bnd_pot = f->n_bnd_pot;
    a.k_rowptr = f->k_rowptr, a.k_col = f->k_col, a.k_val = f->k_val, a.f0 = f->f0;
    a.d = f->d, a.f1 = f->f1, a.ion_den = ion_den, a.potential = node_potential, a.status = status;
    a.t1 = w, a.t2 = w + n, a.t3 = w + 2 * n, a.diag = w + 3 * n, a.x = w + 4 * n, a.r = w + 5 * n;
    a.p = w + 6 * n, a.q = w + 7 * n;
    a.partial_a = w + 8 * n;
    a.partial_b = w + 8 * n + kMaxCoopBlocks;
    a.n0 = c->n0, a.phi0 = c->phi0, a.kte = c->kte, a.qe = c->qe, a.eps0 = c->eps0;
    a.rtol = c->rtol, a.atol = c->atol, a.max_iter = c->max_iter;
    if (f->n_diag < 0 || f->n_diag > OPPB_FIELD_MAX_DIAG || (f->n_diag > 0 && !f->dia_val)) return OPPB_ERR_ARG;
    a.n_diag = f->n_diag;
    for (int j = 0; j < OPPB_FIELD_MAX_DIAG; j++) a.dia_off[j] = f->dia_off[j];
    a.dia_val = f->dia_val;
    CgPlan plan;
    int32_t lo = 0, hi = 0;
    int rc = make_cg_plan(a, options->no_cluster != 0, &plan, &lo, &hi);
    if (rc) return rc;
    if (plan.rows) return solve_by_diagonals(a, plan, lo, hi, options->max_polls, as_stream(stream));
    int blocks = 0;
    if ((rc = coop_grid(&blocks))) return rc;
    void* args[] = {&a};
    if (cudaLaunchCooperativeKernel((const void*)field_newton_kernel, dim3(blocks), dim3(kFieldBlock), args, 0,
                                    as_stream(stream)) != cudaSuccess)
        return OPPB_ERR_LAUNCH;
    count_launches(1);
    return launch_status();
}

extern "C" int oppb_field_solve(const oppb_field_device* f, const oppb_field_consts* c, const double* ion_den,
                                double* node_potential, oppb_field_status* status, void* stream) {
    const oppb_field_options options{OPPB_FIELD_MAX_POLLS, 0};
    return oppb_field_solve_ex(f, c, ion_den, node_potential, status, &options, stream);
}
