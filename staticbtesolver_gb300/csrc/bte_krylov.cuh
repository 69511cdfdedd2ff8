// bte_krylov.cuh -- BiCGSTAB with one thread-block cluster per system.
//
// The iteration of the phase kernels of bte_kernels.cuh (k_bicg_p ..
// k_bicg_x) in one launch: the cluster keeps a system on chip (r, p, q, t in
// registers; x, r_hat, the operator's coefficients and the exchanged vector in
// shared memory, a neighbour's value read from its owner's shared memory), and
// cluster barriers take the place of launches.
//
// What bounds it.  The phase kernels take five launches per iteration of the
// slowest system: on small meshes an iteration is 5 x ~10 us of launch and
// load latency, on large ones the launches go on for the few systems that
// converge last, and every iteration reads 25 vector words per cell.  Here a
// converged system frees its SMs for the next one, and what is left is the
// FP64 pipe.  Measured on GB300: one FP64 instruction of a warp occupies the
// SM's pipe for 19 cycles whatever its active lanes, a dependent one returns
// after 64, a division after 565; a cluster barrier costs 380 cycles, a remote
// shared-memory load 270, a block barrier 34.  So the kernel counts FP64
// instructions:
//  * M (Jacobi) and k_b are folded into the off-diagonal coefficients once per
//    solve (A M = I + C, C[c][f] = k_b fc[f] / D[nb f]) and only inflow faces
//    are kept (SLOTS: 2 on triangles, 3 on tetrahedra): a product costs SLOTS
//    instead of F + 1 operations and needs no p_hat = M p, z = M s; x is
//    accumulated as M^-1 x and scaled once at the end.  2D: 15 operations per
//    cell and iteration instead of 21 (3D: 17 instead of 23);
//  * a block's partial sums are transposed through shared memory, so one warp
//    adds them in 8 + 5 instructions instead of 8 warps in 5 each and 8 more;
//  * one warp per CTA forms the iteration's scalars.
// Solves measured, phase kernels -> clusters: 578 triangles x 32 directions to
// margin 1e-5, 135 -> 17.4 ms; 750 tetrahedra x 128 directions, 228 -> 43 ms;
// 10,082 triangles x 256 systems in mixed precision, three outer iterations, 157
// -> 25 ms (FP64 beyond 4,096 cells keeps the phase kernels, batch_len).  One CSR
// system from host arrays, to 1e-12: 968 unknowns 2.8 -> 0.56 ms, 9,800 unknowns
// 10.0 -> 1.9 ms (9 us a step: 3.7 of the FP64 pipe, the rest barriers and remote
// loads), 32,768 unknowns 20.5 -> 5.6 ms.
// Sums are taken in a fixed order (threads, warps, CTAs), so a solve is
// reproducible to the bit; they are grouped differently from the phase
// kernels', so the two agree to rounding.  The FP64 pipe of the SMs with a CTA is
// 50 % busy on 578 triangles, 54 % on 750 tetrahedra, 43 % in FP32 on 10,082
// triangles (the scalars and sums); barriers and shared-memory latency are the rest.
#pragma once
#include "bte_kernels.cuh"

namespace bte {

constexpr int KC_CTAS = 16;              // CTAs per cluster at most (above 8: opt-in)
constexpr int KC_ROWS = 8;               // cells per thread at most
constexpr int KC_CELLS = THREADS * KC_ROWS;  // cells per CTA at most

struct ClusterSolve {
    int* done;        // [S] as BicgState
    int* iters;       // [S]
    const int* skip;  // [S] nonzero: no solve (done = 4), or nullptr
    int n, len;       // cells, cells per CTA
    double tol;
    int maxit, cycles, track_from;  // as BicgState
    int best;         // nonzero: keep the iterate with the smallest residual (BicgVecs::xb)
};

__device__ __forceinline__ unsigned cluster_rank() {
    unsigned r;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
}
__device__ __forceinline__ unsigned cluster_ctas() {
    unsigned r;
    asm volatile("mov.u32 %0, %%cluster_nctarank;" : "=r"(r));
    return r;
}
// Every thread of every CTA of the cluster; shared-memory writes made before it
// are visible to all of them after it.
__device__ __forceinline__ void cluster_barrier(unsigned ctas) {
    if (ctas == 1) {
        __syncthreads();
        return;
    }
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// Address of this CTA's shared-memory address a in CTA rank of the cluster.
__device__ __forceinline__ unsigned cluster_map(unsigned a, unsigned rank) {
    unsigned r;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(rank));
    return r;
}
__device__ __forceinline__ void cluster_store(unsigned a, double v) {
    asm volatile("st.shared::cluster.f64 [%0], %1;" ::"r"(a), "d"(v) : "memory");
}
// A value at a cluster address (38 cycles in this CTA's own shared memory, 29
// for a plain load; volatile, so the barriers keep their place among them).
__device__ __forceinline__ void cluster_load(unsigned a, double& v) {
    asm volatile("ld.shared::cluster.f64 %0, [%1];" : "=d"(v) : "r"(a));
}
__device__ __forceinline__ void cluster_load(unsigned a, float& v) {
    asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v) : "r"(a));
}

// Dynamic shared memory of k_bicg_cluster for len cells per CTA: the exchanged
// vector, x, r_hat, (best iterate); SLOTS coefficients and neighbour places
// per cell.
template <typename T>
__host__ __device__ constexpr int cluster_row_group() { return sizeof(T) == 4 ? 4 : 1; }
template <typename T>
__host__ __device__ constexpr int cluster_cells(int len) {
    constexpr int g = THREADS * cluster_row_group<T>();
    return (len + g - 1) / g * g;
}
template <typename T>
constexpr size_t cluster_smem_bytes(int len, int slots, bool best) {
    const size_t cells = cluster_cells<T>(len);
    return cells * (sizeof(T) * (3 + (best ? 1 : 0) + slots) + sizeof(uint32_t) * slots);
}

// One system per cluster (y = blockIdx.x / CTAs of the cluster) of
// ceil(n / len) CTAs, len <= KC_CELLS a multiple of 32.  rhs: [S][Np]; the solution goes to op.x_of(y), the outcome to
// done and iters.  SLOTS >= the largest number of nonzero fc of a cell, or of
// entries of a row for a CSR operator.  MINB: CTAs per SM the registers are
// limited for.
template <typename Op>
constexpr bool cluster_csr = false;
template <>
inline constexpr bool cluster_csr<CsrOp> = true;
#define BTE_CLUSTER_ROWS(k)                                        \
    _Pragma("unroll") for (int _g = 0; _g < KC_ROWS / G && _g < groups; ++_g) \
        _Pragma("unroll") for (int _r = 0, k = _g * G; _r < G; ++_r, ++k)

template <typename Op, typename T, int SLOTS, int MINB>
__global__ void __launch_bounds__(THREADS, MINB) k_bicg_cluster(Op op, const T* __restrict__ rhs, size_t Np,
                                                               ClusterSolve st) {
    extern __shared__ __align__(16) unsigned char kc_smem[];
    __shared__ double red[2][THREADS];   // a block's partials of up to two sums
    __shared__ double part[6][2 * KC_CTAS];  // [sum][CTA, half]
    __shared__ struct {
        double a, b, rho, ratio;
        int act, improved;
    } sc;
    enum { RR = 0, RWR = 1, RWQ = 2, TS = 3, TT = 4, RWR2 = 5 };  // RWR2: r_hat.r of a restart
    enum { GO = 0, RESTART = 1, FINISH = 2 };
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const unsigned ctas = cluster_ctas(), rank = cluster_rank();
    const int y = (int)(blockIdx.x / ctas);
    const int first = (int)rank * st.len;                          // this CTA's cells: first + [0, mine)
    const int mine = max(0, min(st.len, st.n - first));
    const int cells = cluster_cells<T>(st.len);                    // slots of the arrays below
    const bool lead = rank == 0 && tid == 0;
    T* sv = reinterpret_cast<T*>(kc_smem);  // the exchanged vector: p, then s
    T* sx = sv + cells;                     // M^-1 x
    T* srw = sx + cells;
    T* sxb = srw + cells;                   // with st.best
    T* scf = sxb + (st.best ? cells : 0);   // [row][SLOTS][THREADS] coefficients of A M
    uint32_t* sat = reinterpret_cast<uint32_t*>(scf + (size_t)SLOTS * cells);  // ... the neighbours' places
    T* xout = op.x_of(y);
    // a warp's rows of 32 cells are taken in groups of G, without a branch
    // inside a group so their loads overlap: the ones with a cell in it.  FP64
    // takes single rows (a row without cells would still fill the pipe).
    constexpr int G = cluster_row_group<T>();
    const int groups = warp * 32 < mine ? (mine - warp * 32 + G * THREADS - 1) / (G * THREADS) : 0;
    if (st.skip && st.skip[y]) {  // the whole cluster leaves together
        if (lead) {
            st.done[y] = 4;
            st.iters[y] = 0;
        }
        return;
    }
    const T* b = rhs + (size_t)y * Np;
    const unsigned sv_a = (unsigned)__cvta_generic_to_shared(sv);
    // cluster address of cell c's value of the exchanged vector
    auto place = [&](int c) {
        const unsigned r = (unsigned)c / (unsigned)st.len;
        return cluster_map(sv_a + (unsigned)sizeof(T) * ((unsigned)c - r * (unsigned)st.len), r);
    };
    const unsigned part_a = (unsigned)__cvta_generic_to_shared(&part[0][0]);

    // Up to two sums (kinds k0, k1 or k1 < 0): every thread's partial, added
    // per block by warps 0 and 1 (k0) and 2 and 3 (k1), each four threads of a
    // column in order and a butterfly, and published to every CTA.  The parts
    // are complete after the cluster barrier at its end.
    auto publish = [&](T v0, T v1, int k0, int k1) {
        red[0][tid] = (double)v0;
        if (k1 >= 0) red[1][tid] = (double)v1;
        __syncthreads();
        const int kind = warp < 2 ? k0 : warp < 4 ? k1 : -1;
        if (kind >= 0) {
            const double* col = red[warp >> 1] + (warp & 1) * 128 + lane;
            double s = col[0];
            s += col[32];
            s += col[64];
            s += col[96];
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
            const unsigned at = (unsigned)(kind * 2 * KC_CTAS) + 2u * rank + (unsigned)(warp & 1);
            if (ctas == 1) {
                if (lane == 0) (&part[0][0])[at] = s;
            } else if (lane < (int)ctas) {
                cluster_store(cluster_map(part_a + 8u * at, (unsigned)lane), s);
            }
        }
        cluster_barrier(ctas);
    };
    int span = 2;  // parts rounded up to a power of two
    while (span < 2 * (int)ctas) span <<= 1;
    // a published sum over its parts, in every lane
    auto total = [&](int kind) {
        const int i = lane & (span - 1);
        double s = i < 2 * (int)ctas ? part[kind][i] : 0.0;
        for (int o = span >> 1; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
        return s;
    };
    // two of them: in one pass while a sum's parts fit in half a warp
    auto totals = [&](int ka, int kb, double& a, double& b) {
        if (span > 16) {
            a = total(ka);
            b = total(kb);
            return;
        }
        const int i = lane & (span - 1);
        double s = i < 2 * (int)ctas ? part[lane < 16 ? ka : kb][i] : 0.0;
        for (int o = span >> 1; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
        a = __shfl_sync(0xffffffffu, s, 0);
        b = __shfl_sync(0xffffffffu, s, 16);
    };
    // (A M v)[c] of row k, v exchanged (face flux: the diagonal of A M is 1)
    auto product = [&](int k, T v) {
        T x[SLOTS], s = cluster_csr<Op> ? (T)0 : v;
#pragma unroll
        for (int f = 0; f < SLOTS; ++f) cluster_load(sat[(k * SLOTS + f) * THREADS + tid], x[f]);
#pragma unroll
        for (int f = 0; f < SLOTS; ++f) s = fmat(scf[(k * SLOTS + f) * THREADS + tid], x[f], s);
        return s;
    };

    T r[KC_ROWS], p[KC_ROWS], q[KC_ROWS], t[KC_ROWS];
    if (ctas > 1) cluster_barrier(ctas);  // every CTA has started: its shared memory may be used
    {
        // 1/D of every cell, exchanged once to scale the coefficients
        BTE_CLUSTER_ROWS(k) {
            const int l = k * THREADS + tid;
            sv[l] = l < mine ? (T)op.inv_diag(y, first + l) : (T)0;
        }
        cluster_barrier(ctas);
        // (two loops: sharing one costs the FP32 kernel 3 % by its registers)
        if constexpr (cluster_csr<Op>) {
            BTE_CLUSTER_ROWS(k) {
                const int l = k * THREADS + tid, c = first + l;
                int m = 0;
                if (l < mine)
                    for (int e = op.rowptr[c]; e < op.rowptr[c + 1] && m < SLOTS; ++e, ++m) {
                        const unsigned at = place(op.col[e]);
                        T d;
                        cluster_load(at, d);
                        scf[(k * SLOTS + m) * THREADS + tid] = (T)op.val[e] * d;
                        sat[(k * SLOTS + m) * THREADS + tid] = at;
                    }
                for (; m < SLOTS; ++m) {
                    scf[(k * SLOTS + m) * THREADS + tid] = 0;
                    sat[(k * SLOTS + m) * THREADS + tid] = cluster_map(sv_a + (unsigned)sizeof(T) * (unsigned)l, rank);
                }
            }
        } else {
            int sb, sd;
            op.bd(y, sb, sd);
            const T kb = op.kb[sb];
            BTE_CLUSTER_ROWS(k) {
                const int l = k * THREADS + tid, c = first + l;
                int m = 0;
                if (l < mine)
                    for (int f = 0; f < op.F; ++f) {
                        const T cf = op.fc[((size_t)sd * op.F + f) * op.Np + c];
                        if (cf == 0) continue;
                        if (m < SLOTS) {
                            const unsigned at = place(op.nb[(size_t)f * op.Np + c]);
                            T d;
                            cluster_load(at, d);
                            scf[(k * SLOTS + m) * THREADS + tid] = kb * cf * d;
                            sat[(k * SLOTS + m) * THREADS + tid] = at;
                        }
                        ++m;
                    }
                for (; m < SLOTS; ++m) {
                    scf[(k * SLOTS + m) * THREADS + tid] = 0;
                    sat[(k * SLOTS + m) * THREADS + tid] = cluster_map(sv_a + (unsigned)sizeof(T) * (unsigned)l, rank);
                }
            }
        }
        T acc = 0;
#pragma unroll
        for (int k = 0; k < KC_ROWS; ++k) r[k] = p[k] = q[k] = t[k] = 0;
        BTE_CLUSTER_ROWS(k) {
            const int l = k * THREADS + tid;
            const T bb = l < mine ? b[first + l] : (T)0;
            r[k] = bb;
            srw[l] = bb;
            if constexpr (sizeof(T) == sizeof(double)) p[k] = bb;  // (FP32 starts from p = 0, see k_bicg_init)
            sx[l] = 0;
            if (st.best) sxb[l] = 0;
            acc = fmat(bb, bb, acc);
        }
        publish(acc, acc, RR, RWR);
    }
    // breakdown restart (bicg_restart_chunk): x = q = p = 0, r = b, r_hat = 6.8 b + 0.6
    auto restart = [&]() {
        T acc = 0;
        BTE_CLUSTER_ROWS(k) {
            const int l = k * THREADS + tid;
            const T bb = l < mine ? b[first + l] : (T)0;
            const T rh = bb * (T)6.8 + (T)0.6;
            sx[l] = 0;
            q[k] = 0;
            p[k] = 0;
            r[k] = bb;
            srw[l] = rh;
            acc = fmat(rh, bb, acc);
        }
        publish(acc, 0, RWR2, -1);
    };
    // Scalars of the iteration, kept by warp 0 of every CTA (the same in all).
    // Norms are compared through their squares (a square root takes 600
    // cycles), all comparisons of a step at once, one per lane (each takes 64);
    // the part of beta known an iteration ahead, (alpha / omega) / rho, is
    // formed by the last warp while the block updates x and r.
    double bestr = 0.0, rho = 1.0, alpha = 1.0, omega = 1.0;
    double rr = 0.0, rr0 = 0.0, stop = 0.0;  // ||r||^2, ||b||^2, its share that ends the solve
    bool flagged = false;   // the last iteration restarted
    if (warp == 0) {
        rr = rr0 = bestr = total(RR);
        stop = st.tol * st.tol * rr0;
        if (lane == 0) sc.ratio = 1.0;
    }
    const bool in_range = stop > 1e-280 && stop < 1e280;  // (warp 0)
    for (int i = 1;; ++i) {
        if (warp == 0) {  // convergence, rho, beta (bicg_p_body)
            const bool fresh = i > 1 && !flagged;
            double rho_new;
            if (fresh) totals(RWR, RR, rho_new, rr);
            else rho_new = total(flagged ? RWR2 : RWR);
            double v = rr, lim = stop;
            if (lane == 1) lim = 1e-100;
            if (lane == 2) v = fabs(rho_new), lim = 1e-200;
            if (lane == 3) lim = bestr;
            if (lane == 4) lim = 1.0e300;
            const unsigned below = __ballot_sync(0xffffffffu, v < lim);
            int act = GO, code = 0, its = i - 1;
            bool improved = false;
            double beta = 0.0;
            // (squares that under- or overflow: the norms themselves)
            if (fresh && (in_range ? (below & 1u) != 0 : sqrt(rr) / sqrt(rr0) < st.tol)) {
                act = FINISH;
                code = 1;
            }
            if (act == GO && st.best) {
                improved = fresh && i > st.track_from && (below & 8u);
                if (improved) bestr = rr;
                if (i > st.maxit * st.cycles || !(below & 16u)) {
                    act = FINISH;
                    code = 3;
                }
            } else if (act == GO && i > st.maxit) {
                act = FINISH;
                code = 3;
                its = st.maxit;
            }
            if (act == GO && (below & 2u)) {
                act = FINISH;
                code = 2;
            }
            if (act == GO) {
                flagged = (below & 4u) != 0;
                if (flagged) {
                    act = RESTART;
                    alpha = omega = rho = 1.0;
                    if (lane == 0) sc.ratio = 1.0;
                } else {
                    beta = rho_new * sc.ratio;
                    rho = rho_new;
                }
            }
            if (lane == 0) {
                sc.act = act;
                sc.improved = improved;
                sc.a = act == FINISH ? (double)code : omega;
                sc.b = beta;
            }
            if (act == FINISH && lead) {
                st.done[y] = code;
                st.iters[y] = its;
            }
        }
        __syncthreads();
        const int act = sc.act;
        if (act == FINISH) {
            const T* xs = st.best && sc.a == 3.0 && !sc.improved ? sxb : sx;
#pragma unroll
            for (int k = 0; k < KC_ROWS; ++k) {
                const int l = k * THREADS + tid;
                if (l < mine) xout[first + l] = (T)op.inv_diag(y, first + l) * xs[l];
            }
            // the padding cells of the system stay zero
            for (int c = st.n + (int)rank * THREADS + tid; c < (int)Np; c += (int)ctas * THREADS) xout[c] = 0;
            break;
        }
        if (st.best && sc.improved)
            BTE_CLUSTER_ROWS(k) sxb[k * THREADS + tid] = sx[k * THREADS + tid];
        if (act == RESTART) {
            restart();
            continue;
        }
        {
            const T om = (T)sc.a, bt = (T)sc.b;
            BTE_CLUSTER_ROWS(k) {
                const int l = k * THREADS + tid;
                T u = fmat(-om, q[k], p[k]);
                u = fmat(bt, u, r[k]);
                p[k] = u;
                sv[l] = u;
            }
        }
        cluster_barrier(ctas);
        {  // q = A M p, r_hat . q
            T acc = 0;
            BTE_CLUSTER_ROWS(k) {
                q[k] = product(k, p[k]);
                acc = fmat(srw[k * THREADS + tid], q[k], acc);
            }
            publish(acc, 0, RWQ, -1);
        }
        if (warp == 0) {
            const double temp = total(RWQ);
            alpha = rho / temp;
            flagged = fabs(temp) < 1e-200;
            if (flagged) {
                alpha = omega = rho = 1.0;
                if (lane == 0) {
                    sc.act = RESTART;
                    sc.ratio = 1.0;
                }
            } else if (lane == 0) {
                sc.a = alpha;
                sc.rho = rho;
            }
        }
        __syncthreads();
        if (sc.act == RESTART) {
            restart();
            continue;
        }
        const T al = (T)sc.a;
        BTE_CLUSTER_ROWS(k) {
            const int l = k * THREADS + tid;
            const T s = fmat(-al, q[k], r[k]);
            r[k] = s;
            sv[l] = s;
        }
        cluster_barrier(ctas);
        {  // t = A M s, t . s, t . t
            T a0 = 0, a1 = 0;
            BTE_CLUSTER_ROWS(k) {
                t[k] = product(k, r[k]);
                a0 = fmat(t[k], r[k], a0);
                a1 = fmat(t[k], t[k], a1);
            }
            publish(a0, a1, TS, TT);
        }
        if (warp == 0) {
            double tt, ts;
            totals(TT, TS, tt, ts);
            omega = tt > 0.0 ? ts / tt : 0.0;
            if (lane == 0) sc.b = omega;
        }
        __syncthreads();
        {
            const T om = (T)sc.b;
            if (warp == NWARP - 1) {  // lane 0: alpha / omega, the others: 1 / rho
                const double v = lane == 0 ? sc.a : 1.0, w = lane == 0 ? sc.b : sc.rho;
                const double h = v / w;
                const double ratio = h * __shfl_sync(0xffffffffu, h, 1);
                if (lane == 0) sc.ratio = ratio;
            }
            T a0 = 0, a1 = 0;
            BTE_CLUSTER_ROWS(k) {
                const int l = k * THREADS + tid;
                T u = fmat(al, p[k], sx[l]);
                u = fmat(om, r[k], u);
                sx[l] = u;
                const T rn = fmat(-om, t[k], r[k]);
                r[k] = rn;
                a0 = fmat(rn, rn, a0);
                a1 = fmat(srw[l], rn, a1);
            }
            publish(a0, a1, RR, RWR);
        }
    }
    if (ctas > 1) cluster_barrier(ctas);  // no CTA leaves while another may read its shared memory
}

// Largest number of nonzero inflow coefficients of a cell in any direction.
__global__ void k_max_inflow(const double* __restrict__ fc, int F, int n, size_t Np, int* __restrict__ out) {
    const int c = blockIdx.x * blockDim.x + threadIdx.x;
    const int d = blockIdx.y;
    int m = 0;
    if (c < n)
        for (int f = 0; f < F; ++f) m += fc[((size_t)d * F + f) * Np + c] != 0.0;
    m = __reduce_max_sync(0xffffffffu, m);
    if ((threadIdx.x & 31) == 0 && m > 0) atomicMax(out, m);
}

}  // namespace bte
