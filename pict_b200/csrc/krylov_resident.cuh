// krylov_resident.cuh -- Krylov solves of small systems held on chip by one thread-block cluster (included by
// krylov.cu).
//
// A system of n cells is cut into one contiguous run of ceil(n / CL) cells per CTA of the cluster; thread t of a
// CTA owns the cells t, t + RS_THREADS, ... of the run.  Every vector of the iteration stays in the owner's
// registers, the stencil rows in registers (small runs) or in the owner's shared memory, and the one vector whose
// neighbours are needed is exchanged through a shared-memory buffer per CTA that the whole cluster reads
// (distributed shared memory; each thread keeps the cluster addresses of its cells' neighbours, so connected and
// periodic faces cost nothing extra).  Global memory is read once at the start and written once at the end.
//
// What bounds it: the chain of an iteration (for CG one or two cluster barriers, one remote read, one FP64 reduction),
// not bytes: nothing but the result leaves the SMs.  The sweeping forms (k_cg1_cluster, and k_bicgstab with four grid
// barriers an iteration) send every vector through L2 between barriers: ~5.5 us a CG iteration on up to 32k cells,
// here 1.7 us (4,096 cells) to 2.1 us.  Measured on whole passes: 8 steps of a 64^2 cavity in FP32 6.8 -> 2.8 ms, 2 steps
// of the 27,648-cell street 19.2 -> 6.4 ms, 2 steps of a 32^3 cavity in FP64 5.8 -> 2.8 ms, forward and backward of
// 4 steps on a 128^2 periodic box in FP64 16.1 -> 6.8 ms.
#pragma once

namespace pict {

constexpr int RS_THREADS = 512;
constexpr int RS_NV = 6;  // values per CTA partial

struct ResidentRed {
    double warp[RS_THREADS / 32][RS_NV];
    double part[2][KC_MAX_CL][RS_NV];
};

__device__ __forceinline__ unsigned smem_addr(const void* p) { return (unsigned)__cvta_generic_to_shared(p); }

__device__ __forceinline__ unsigned cluster_addr(unsigned local, int rank) {
    unsigned r;
    asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(local), "r"(rank));
    return r;
}

__device__ __forceinline__ void cluster_load(unsigned addr, float& v) {
    asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v) : "r"(addr));
}

__device__ __forceinline__ void cluster_load(unsigned addr, double& v) {
    asm volatile("ld.shared::cluster.f64 %0, [%1];" : "=d"(v) : "r"(addr));
}

__device__ __forceinline__ void cluster_store(unsigned addr, double v) {
    asm volatile("st.shared::cluster.f64 [%0], %1;" ::"r"(addr), "d"(v) : "memory");
}

__device__ __forceinline__ void cluster_arrive() { asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory"); }
__device__ __forceinline__ void cluster_wait() { asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory"); }
__device__ __forceinline__ void cluster_barrier() {
    cluster_arrive();
    cluster_wait();
}

// Sum of NV values over all threads of the cluster, the same bits in every thread: butterfly in each warp, the
// warps' sums by the first warp, its result pushed into every CTA's table, one cluster barrier, and the CTAs' sums by
// a butterfly in every warp (no second block barrier).  Sum e writes table e & 1: a CTA gets there only after the
// barrier of sum e - 1, which every CTA reaches only after it has read table e - 2.
// In two parts, up to and with the barrier and after it, so that a caller can start the remote reads that the barrier
// made visible before it waits for the sums.
template <int NV>
__device__ __forceinline__ void resident_sum_push(ResidentRed& R, int CL, int rank, unsigned epoch, double (&v)[NV]) {
    static_assert(NV <= RS_NV, "resident_sum: too many values");
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, par = epoch & 1;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
#pragma unroll
        for (int k = 0; k < NV; ++k) v[k] += __shfl_xor_sync(0xffffffffu, v[k], o);
    }
    if (lane == 0) {
#pragma unroll
        for (int k = 0; k < NV; ++k) R.warp[warp][k] = v[k];
    }
    __syncthreads();
    if (warp == 0) {
        double s[NV];
#pragma unroll
        for (int k = 0; k < NV; ++k) s[k] = R.warp[lane & 15][k];
#pragma unroll
        for (int o = 8; o > 0; o >>= 1) {
#pragma unroll
            for (int k = 0; k < NV; ++k) s[k] += __shfl_xor_sync(0xffffffffu, s[k], o);
        }
        if (lane < CL) {
            const unsigned to = cluster_addr(smem_addr(&R.part[par][rank][0]), lane);
#pragma unroll
            for (int k = 0; k < NV; ++k) cluster_store(to + 8 * k, s[k]);
        }
        __syncwarp();
    }
    cluster_barrier();
}

template <int NV>
__device__ __forceinline__ void resident_sum_read(ResidentRed& R, int CL, unsigned epoch, double (&v)[NV]) {
    const int r = threadIdx.x & 15, par = epoch & 1;
#pragma unroll
    for (int k = 0; k < NV; ++k) v[k] = r < CL ? R.part[par][r][k] : 0.0;
#pragma unroll
    for (int o = 8; o > 0; o >>= 1) {
#pragma unroll
        for (int k = 0; k < NV; ++k) v[k] += __shfl_xor_sync(0xffffffffu, v[k], o);
    }
}

template <int NV>
__device__ __forceinline__ void resident_sum(ResidentRed& R, int CL, int rank, unsigned& epoch, double (&v)[NV]) {
    resident_sum_push<NV>(R, CL, rank, epoch, v);
    resident_sum_read<NV>(R, CL, epoch, v);
    ++epoch;
}

__device__ __forceinline__ float fma_rn(float a, float b, float c) { return __fmaf_rn(a, b, c); }
__device__ __forceinline__ double fma_rn(double a, double b, double c) { return __fma_rn(a, b, c); }

// The cells of this thread: stencil rows (registers, or shared memory when ROWS_SMEM) and neighbour addresses.
template <typename T, int D, int CPT, bool ROWS_SMEM>
struct ResidentRows {
    static constexpr int K = 2 * D + 1;
    T reg[ROWS_SMEM ? 1 : CPT * K];
    T* sm;             // [K][CPT * RS_THREADS]
    unsigned nb[CPT][2 * D];

    __device__ __forceinline__ T get(int k, int j) const {
        if constexpr (ROWS_SMEM) return sm[(size_t)j * (CPT * RS_THREADS) + k * RS_THREADS + threadIdx.x];
        else return reg[k * K + j];
    }
    __device__ __forceinline__ void set(int k, int j, T v) {
        if constexpr (ROWS_SMEM) sm[(size_t)j * (CPT * RS_THREADS) + k * RS_THREADS + threadIdx.x] = v;
        else reg[k * K + j] = v;
    }
    // cells [c0, c0 + n) of the system, `run` per CTA, this CTA holds [first, first + cnt); a missing neighbour
    // reads the cell itself with coefficient 0 (as spmv_row masks it); cells beyond cnt read slot 0 of the buffer
    __device__ __forceinline__ void load(const pict_domain_t& dom, const T* __restrict__ coef, bool trans, int c0, int run,
                                         int first, int cnt, int rank, unsigned buf) {
        const int N = dom.num_cells;
#pragma unroll
        for (int k = 0; k < CPT; ++k) {
            const int l = k * RS_THREADS + threadIdx.x;
            const bool own = l < cnt;
            const int i = first + (own ? l : 0);
            set(k, 0, own ? coef[i] : T(0));
            const unsigned self = cluster_addr(buf + (unsigned)sizeof(T) * (own ? l : 0), rank);
            const pict_block_t& B = dom.blocks[dom.cell_block[i]];
            int q[3];
            unflatten(i - B.offset, B.size, q);
            const int stride[3] = {1, B.size[0], B.size[0] * B.size[1]};
#pragma unroll
            for (int f = 0; f < 2 * D; ++f) {
                int j = i + ((f & 1) ? stride[f >> 1] : -stride[f >> 1]);
                int back = f ^ 1;
                if (at_face(q, B.size, f)) {
                    j = dom.nbr[(size_t)f * N + i];
                    if (B.face[f].type == PICT_FACE_CONNECTED) back = B.face[f].conn_axes[0];
                }
                const bool ok = own && j >= 0;
                set(k, f + 1, ok ? (trans ? coef[(size_t)(back + 1) * N + j] : coef[(size_t)(f + 1) * N + i]) : T(0));
                const int g = ok ? j - c0 : 0;
                const int r = g / run;
                nb[k][f] = ok ? cluster_addr(buf + (unsigned)sizeof(T) * (g - r * run), r) : self;
            }
        }
    }
    // row k applied to the exchanged vector, whose value at the cell itself is `self` (spmv_row's order of terms)
    __device__ __forceinline__ T apply(int k, T self, unsigned shift = 0) const {
        T v[2 * D];
#pragma unroll
        for (int f = 0; f < 2 * D; ++f) cluster_load(nb[k][f] + shift, v[f]);
        T acc = get(k, 0) * self;
#pragma unroll
        for (int f = 0; f < 2 * D; ++f) acc += get(k, f + 1) * v[f];
        return acc;
    }
    // the same with the neighbours' values formed as v + bt * q from two exchanged vectors `qshift` bytes apart
    __device__ __forceinline__ T apply2(int k, T self, unsigned shift, unsigned qshift, T bt) const {
        T v[2 * D], q[2 * D];
#pragma unroll
        for (int f = 0; f < 2 * D; ++f) {
            cluster_load(nb[k][f] + shift, v[f]);
            cluster_load(nb[k][f] + shift + qshift, q[f]);
        }
        T acc = get(k, 0) * self;
#pragma unroll
        for (int f = 0; f < 2 * D; ++f) acc += get(k, f + 1) * (v[f] + bt * q[f]);
        return acc;
    }
};

// shared memory of a resident solve: NBUF exchange buffers of one run, the rows if they live there
template <typename T, int D, int CPT, bool ROWS_SMEM>
constexpr size_t resident_smem(int nbuf) {
    return sizeof(T) * (size_t)CPT * RS_THREADS * (nbuf + (ROWS_SMEM ? 2 * D + 1 : 0));
}

// CG, single-reduction recurrence (k_cg1): the iterates, stopping rule and reports of k_cg1_cluster.  COPIES: every
// thread also carries r and s of its cells' neighbours and advances them with the neighbours' w, so an iteration needs
// one cluster barrier (w and the sums together) instead of two (r, then the sums), for 4 D more values per cell.
template <typename T, int D, int CPT, bool ROWS_SMEM, bool COPIES>
__global__ void __launch_bounds__(RS_THREADS, 1) k_cg1_resident(KArgs<T> a, bool trans) {
    extern __shared__ __align__(16) unsigned char rs_smem[];
    __shared__ ResidentRed R;
    const pict_domain_t& dom = a.dom;
    cgrp::cluster_group cl = cgrp::this_cluster();
    const int CL = (int)cl.num_blocks(), rank = (int)cl.block_rank();
    T* buf = reinterpret_cast<T*>(rs_smem);
    constexpr unsigned WS = sizeof(T) * CPT * RS_THREADS;  // byte distance of the second exchange buffer (COPIES)
    ResidentRows<T, D, CPT, ROWS_SMEM> A;
    A.sm = buf + (COPIES ? 2 : 1) * CPT * RS_THREADS;
    unsigned epoch = 0;
    cluster_barrier();  // every CTA runs before any distributed shared memory access

    // the systems of this cluster: a fixed share (they are ordered largest first), so a solve is one launch that needs
    // no cleared counter and writes every report itself
    for (int sys = blockIdx.x / CL; sys < dom.num_sims; sys += gridDim.x / CL) {
        const int c0 = dom.sim_cells[sys], n = dom.sim_cells[sys + 1] - c0;
        const int run = (n + CL - 1) / CL;
        const int first = min(c0 + rank * run, c0 + n), cnt = min(run, c0 + n - first);
        // a CTA without cells (n < rank * run) reads cell c0 with zero coefficients and contributes nothing
        A.load(dom, a.coef, trans, c0, run, cnt > 0 ? first : c0, cnt, rank, smem_addr(buf));
        T r[CPT], s[CPT], p[CPT], x[CPT], w[CPT];
        double acc[3] = {0.0, 0.0, 0.0};
#pragma unroll
        for (int k = 0; k < CPT; ++k) {
            const int l = k * RS_THREADS + threadIdx.x;
            const bool own = l < cnt;
            r[k] = own ? a.b[first + l] : T(0);
            x[k] = own && !a.x_zero ? a.x[first + l] : T(0);
            s[k] = p[k] = T(0);
            acc[2] += (double)r[k] * (double)r[k];
        }
        if (!a.x_zero) {  // r0 = b - A x0
#pragma unroll
            for (int k = 0; k < CPT; ++k) buf[k * RS_THREADS + threadIdx.x] = x[k];
            cluster_barrier();
#pragma unroll
            for (int k = 0; k < CPT; ++k) r[k] -= A.apply(k, x[k]);
            cluster_barrier();
        }
#pragma unroll
        for (int k = 0; k < CPT; ++k) buf[k * RS_THREADS + threadIdx.x] = r[k];
        cluster_barrier();
        T rn[COPIES ? CPT : 1][2 * D], sn[COPIES ? CPT : 1][2 * D], wn[COPIES ? CPT : 1][2 * D];
#pragma unroll
        for (int k = 0; k < CPT; ++k) {
            if constexpr (COPIES) {  // the neighbours' r0, and w0 into the second buffer
                w[k] = A.get(k, 0) * r[k];
#pragma unroll
                for (int f = 0; f < 2 * D; ++f) {
                    cluster_load(A.nb[k][f], rn[k][f]);
                    sn[k][f] = T(0);
                    w[k] += A.get(k, f + 1) * rn[k][f];
                }
                buf[(CPT + k) * RS_THREADS + threadIdx.x] = w[k];
            } else {
                w[k] = A.apply(k, r[k]);
            }
            acc[0] += (double)r[k] * (double)r[k];
            acc[1] += (double)w[k] * (double)r[k];
        }
        resident_sum<3>(R, CL, rank, epoch, acc);
        if constexpr (COPIES) {
#pragma unroll
            for (int k = 0; k < CPT; ++k)
#pragma unroll
                for (int f = 0; f < 2 * D; ++f) cluster_load(A.nb[k][f] + WS, wn[k][f]);
        }
        pict_solve_info_t inf = fresh_info();
        // crit < tol is tested as g' < tol^2 (n), which keeps a root and a division out of the iteration's chain (at
        // least the smallest positive number, so that a residual of exactly 0 stops the tiniest tolerance too)
        double g = acc[0], alpha = acc[0] / acc[1], beta = 0.0, gn = acc[0];
        const double stop = a.tol > 0.0 ? fmax(a.tol * a.tol * (a.normalized ? (double)n : 1.0), 4.9406564584124654e-324) : -1.0;
        bool active = true;
        if (acc[2] == 0.0) {
            inf.converged = 1;
            inf.used_iterations = 0;
            active = false;
#pragma unroll
            for (int k = 0; k < CPT; ++k) x[k] = T(0);
        }
        for (int it = 0; active && it < a.maxit; ++it) {
            const T al = (T)alpha, bt = (T)beta;
            double d[2] = {0.0, 0.0};
            if constexpr (COPIES) {
                // this thread's copies of the neighbours' s and r advance as their owners advance them (the same
                // operations on the same values), so only w travels, together with the sums
                const unsigned to = (it & 1) ? WS : 0u;
#pragma unroll
                for (int k = 0; k < CPT; ++k) {
                    p[k] = fma_rn(bt, p[k], r[k]);
                    s[k] = fma_rn(bt, s[k], w[k]);
                    r[k] = fma_rn(-al, s[k], r[k]);
                    T acc_w = A.get(k, 0) * r[k];
#pragma unroll
                    for (int f = 0; f < 2 * D; ++f) {
                        sn[k][f] = fma_rn(bt, sn[k][f], wn[k][f]);
                        rn[k][f] = fma_rn(-al, sn[k][f], rn[k][f]);
                        acc_w += A.get(k, f + 1) * rn[k][f];
                    }
                    w[k] = acc_w;
                    buf[(to ? CPT * RS_THREADS : 0) + k * RS_THREADS + threadIdx.x] = w[k];
                    d[0] += (double)r[k] * (double)r[k];
                    d[1] += (double)w[k] * (double)r[k];
                }
                resident_sum_push<2>(R, CL, rank, epoch, d);
#pragma unroll
                for (int k = 0; k < CPT; ++k)
#pragma unroll
                    for (int f = 0; f < 2 * D; ++f) cluster_load(A.nb[k][f] + to, wn[k][f]);
#pragma unroll
                for (int k = 0; k < CPT; ++k) x[k] = fma_rn(al, p[k], x[k]);
                resident_sum_read<2>(R, CL, epoch, d);
                ++epoch;
            } else {
#pragma unroll
                for (int k = 0; k < CPT; ++k) {
                    p[k] = r[k] + bt * p[k];
                    s[k] = w[k] + bt * s[k];
                    r[k] -= al * s[k];
                    buf[k * RS_THREADS + threadIdx.x] = r[k];
                }
                cluster_arrive();
#pragma unroll
                for (int k = 0; k < CPT; ++k) {
                    x[k] += al * p[k];
                    d[0] += (double)r[k] * (double)r[k];
                }
                cluster_wait();
#pragma unroll
                for (int k = 0; k < CPT; ++k) {
                    w[k] = A.apply(k, r[k]);
                    d[1] += (double)w[k] * (double)r[k];
                }
                resident_sum<2>(R, CL, rank, epoch, d);
            }
            gn = d[0];
            inf.used_iterations = it;
            if (!isfinite(gn)) { inf.finite = 0; active = false; }
            else if (gn < stop) { inf.converged = 1; active = false; }
            else {
                beta = gn / g;
                alpha = gn / (d[1] - beta * gn / alpha);
                g = gn;
            }
        }
        if (inf.used_iterations >= 0 && acc[2] != 0.0) inf.final_residual = conv_crit(gn, a.normalized, n);
        T mean = T(0);
        if (a.sub_mean) {
            double m[1] = {0.0};
#pragma unroll
            for (int k = 0; k < CPT; ++k) m[0] += (double)x[k];
            resident_sum<1>(R, CL, rank, epoch, m);
            mean = (T)(m[0] / (double)n);
        }
#pragma unroll
        for (int k = 0; k < CPT; ++k) {
            const int l = k * RS_THREADS + threadIdx.x;
            if (l >= cnt) continue;
            const int i = first + l;
            const T v = x[k] - mean;
            a.x[i] = v;
            if (a.write_bp) {
                const pict_block_t& B = dom.blocks[dom.cell_block[i]];
                reinterpret_cast<T*>(B.pressure)[i - B.offset] = v;
            }
        }
        if (rank == 0 && threadIdx.x == 0) a.info[sys] = inf;
        __syncwarp();
        cluster_barrier();  // every CTA is done with the buffers and the tables of this system
    }
}

// BiCGStab (k_bicgstab: the same iterates, per-component stopping rule and reports) with four cluster barriers per
// iteration.  Exchange buffers: X[c] holds r' (then s), Q[c] holds p - omega v, so a neighbour's new search
// direction r' + beta (p - omega v) is formed by the reader once beta is known and needs no barrier of its own.
template <typename T, int D, int NR, int CPT, bool ROWS_SMEM>
__global__ void __launch_bounds__(RS_THREADS, 1) k_bicgstab_resident(KArgs<T> a, bool trans) {
    static_assert(2 * NR <= RS_NV, "too many right-hand sides per launch");
    extern __shared__ __align__(16) unsigned char rs_smem[];
    __shared__ ResidentRed R;
    constexpr int RUN = CPT * RS_THREADS;
    constexpr unsigned XS = sizeof(T) * RUN;          // byte distance from X[c] to X[c + 1]
    constexpr unsigned QS = sizeof(T) * RUN * NR;     // byte distance from X[c] to Q[c]
    const pict_domain_t& dom = a.dom;
    const size_t NS = (size_t)dom.num_cells;
    cgrp::cluster_group cl = cgrp::this_cluster();
    const int CL = (int)cl.num_blocks(), rank = (int)cl.block_rank();
    T* buf = reinterpret_cast<T*>(rs_smem);
    T* bufq = buf + RUN * NR;
    ResidentRows<T, D, CPT, ROWS_SMEM> A;
    A.sm = buf + 2 * RUN * NR;
    unsigned epoch = 0;
    cluster_barrier();  // every CTA runs before any distributed shared memory access

    // the systems of this cluster: a fixed share (they are ordered largest first), so a solve is one launch that needs
    // no cleared counter and writes every report itself
    for (int sys = blockIdx.x / CL; sys < dom.num_sims; sys += gridDim.x / CL) {
        const int c0 = dom.sim_cells[sys], n = dom.sim_cells[sys + 1] - c0;
        const int run = (n + CL - 1) / CL;
        const int first = min(c0 + rank * run, c0 + n), cnt = min(run, c0 + n - first);
        A.load(dom, a.coef, trans, c0, run, cnt > 0 ? first : c0, cnt, rank, smem_addr(buf));
        T r[CPT][NR], rw[CPT][NR], p[CPT][NR], v[CPT][NR], x[CPT][NR], t[CPT][NR];
        double rwr[NR], rho[NR], alpha[NR], omega[NR];
        double sum[2 * NR];
        unsigned act = 0;
        pict_solve_info_t inf[NR];
#pragma unroll
        for (int c = 0; c < 2 * NR; ++c) sum[c] = 0.0;
#pragma unroll
        for (int k = 0; k < CPT; ++k) {
            const int l = k * RS_THREADS + threadIdx.x;
            const bool own = l < cnt;
#pragma unroll
            for (int c = 0; c < NR; ++c) {
                r[k][c] = own ? a.b[c * NS + first + l] : T(0);
                x[k][c] = own && !a.x_zero ? a.x[c * NS + first + l] : T(0);
                p[k][c] = v[k][c] = T(0);
                sum[NR + c] += (double)r[k][c] * (double)r[k][c];
            }
        }
        if (!a.x_zero) {  // r = b - A x
#pragma unroll
            for (int k = 0; k < CPT; ++k)
#pragma unroll
                for (int c = 0; c < NR; ++c) buf[c * RUN + k * RS_THREADS + threadIdx.x] = x[k][c];
            cluster_barrier();
#pragma unroll
            for (int k = 0; k < CPT; ++k)
#pragma unroll
                for (int c = 0; c < NR; ++c) r[k][c] -= A.apply(k, x[k][c], c * XS);
            cluster_barrier();
        }
#pragma unroll
        for (int k = 0; k < CPT; ++k)
#pragma unroll
            for (int c = 0; c < NR; ++c) {
                rw[k][c] = r[k][c];
                sum[c] += (double)r[k][c] * (double)r[k][c];
                buf[c * RUN + k * RS_THREADS + threadIdx.x] = r[k][c];
                bufq[c * RUN + k * RS_THREADS + threadIdx.x] = T(0);
            }
        resident_sum<2 * NR>(R, CL, rank, epoch, sum);
#pragma unroll
        for (int c = 0; c < NR; ++c) {
            inf[c] = fresh_info();
            rho[c] = alpha[c] = omega[c] = 0.0;
            rwr[c] = sum[c];
            if (sum[NR + c] == 0.0) {
                inf[c].converged = 1;
                inf[c].used_iterations = 0;
#pragma unroll
                for (int k = 0; k < CPT; ++k) x[k][c] = T(0);
            } else {
                const double crit = conv_crit(sum[c], a.normalized, n);
                if (crit < a.tol) {
                    inf[c].converged = 1;
                    inf[c].final_residual = crit;
                } else {
                    act |= 1u << c;
                }
            }
        }
        for (int it = 0; act && it < a.maxit; ++it) {
            // p = r + beta (p - omega v), v = A p, rw.v
            double d1[NR];
#pragma unroll
            for (int c = 0; c < NR; ++c) {
                d1[c] = 0.0;
                if (!((act >> c) & 1u)) continue;
                const double beta = it > 0 ? (rwr[c] / rho[c]) * (alpha[c] / omega[c]) : 0.0;
                rho[c] = rwr[c];
                const T bt = (T)beta, om = (T)omega[c];
#pragma unroll
                for (int k = 0; k < CPT; ++k) {
                    p[k][c] = r[k][c] + bt * (p[k][c] - om * v[k][c]);
                    v[k][c] = A.apply2(k, p[k][c], c * XS, QS, bt);
                    d1[c] += (double)rw[k][c] * (double)v[k][c];
                }
            }
            resident_sum<NR>(R, CL, rank, epoch, d1);
            // s = r - alpha v, x += alpha p, |s|^2
            double d2[NR];
#pragma unroll
            for (int c = 0; c < NR; ++c) {
                if (!((act >> c) & 1u)) { d2[c] = 0.0; continue; }
                alpha[c] = rho[c] / d1[c];
                d2[c] = 0.0;
                const T al = (T)alpha[c];
#pragma unroll
                for (int k = 0; k < CPT; ++k) {
                    r[k][c] = r[k][c] - al * v[k][c];
                    x[k][c] = x[k][c] + al * p[k][c];
                    buf[c * RUN + k * RS_THREADS + threadIdx.x] = r[k][c];
                    d2[c] += (double)r[k][c] * (double)r[k][c];
                }
            }
            resident_sum<NR>(R, CL, rank, epoch, d2);
#pragma unroll
            for (int c = 0; c < NR; ++c) {
                if (!((act >> c) & 1u)) continue;
                const double nr = conv_crit(d2[c], a.normalized, n);
                inf[c].used_iterations = it;
                inf[c].final_residual = nr;
                if (!isfinite(nr)) { inf[c].finite = 0; act &= ~(1u << c); }
                else if (nr < a.tol) { inf[c].converged = 1; act &= ~(1u << c); }
            }
            if (!act) break;
            // t = A s, t.s, t.t
            double d3[2 * NR];
#pragma unroll
            for (int c = 0; c < NR; ++c) {
                d3[2 * c] = d3[2 * c + 1] = 0.0;
                if (!((act >> c) & 1u)) continue;
#pragma unroll
                for (int k = 0; k < CPT; ++k) {
                    t[k][c] = A.apply(k, r[k][c], c * XS);
                    d3[2 * c] += (double)t[k][c] * (double)r[k][c];
                    d3[2 * c + 1] += (double)t[k][c] * (double)t[k][c];
                }
            }
            resident_sum<2 * NR>(R, CL, rank, epoch, d3);
            // x += omega s, r = s - omega t, r.r, rw.r
            double d4[2 * NR];
#pragma unroll
            for (int c = 0; c < NR; ++c) {
                d4[2 * c] = d4[2 * c + 1] = 0.0;
                if (!((act >> c) & 1u)) continue;
                omega[c] = d3[2 * c] / d3[2 * c + 1];
                const T om = (T)omega[c];
#pragma unroll
                for (int k = 0; k < CPT; ++k) {
                    x[k][c] = x[k][c] + om * r[k][c];
                    r[k][c] = r[k][c] - om * t[k][c];
                    buf[c * RUN + k * RS_THREADS + threadIdx.x] = r[k][c];
                    bufq[c * RUN + k * RS_THREADS + threadIdx.x] = p[k][c] - om * v[k][c];
                    d4[2 * c] += (double)r[k][c] * (double)r[k][c];
                    d4[2 * c + 1] += (double)rw[k][c] * (double)r[k][c];
                }
            }
            resident_sum<2 * NR>(R, CL, rank, epoch, d4);
#pragma unroll
            for (int c = 0; c < NR; ++c) {
                if (!((act >> c) & 1u)) continue;
                rwr[c] = d4[2 * c + 1];
                const double nr = conv_crit(d4[2 * c], a.normalized, n);
                inf[c].final_residual = nr;
                if (nr < a.tol) {
                    inf[c].converged = 1;
                    inf[c].used_iterations = it + 1;
                    act &= ~(1u << c);
                }
            }
        }
#pragma unroll
        for (int k = 0; k < CPT; ++k) {
            const int l = k * RS_THREADS + threadIdx.x;
            if (l >= cnt) continue;
#pragma unroll
            for (int c = 0; c < NR; ++c) a.x[c * NS + first + l] = x[k][c];
        }
        if (rank == 0 && threadIdx.x == 0) {
#pragma unroll
            for (int c = 0; c < NR; ++c) a.info[sys * a.nrhs + c] = inf[c];
        }
        __syncwarp();
        cluster_barrier();  // every CTA is done with the buffers and the tables of this system
    }
}

}  // namespace pict
