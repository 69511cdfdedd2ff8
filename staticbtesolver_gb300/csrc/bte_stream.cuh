// bte_stream.cuh -- the upwind sweep as a stream of positions (k_sweep_stream).
//
// The substitution of k_sweep (bte_transport.cuh), with everything that does
// not depend on the solution brought to shared memory ahead of its use.
//
// What bounds it.  k_sweep's levels wait on memory: the cell-addressed loads
// (an L2 round trip each level), the second round of a level wider than the
// block (three dependent loads, none ahead), and above all upstream values too
// old for the block's ring, two dependent loads in a third to a half of the
// levels.  A level of 118 cells took ~3,600 cycles on a square of 100,352
// triangles.  What is left here is the FP64 pipe and, for narrow levels, the
// chain of barrier, shared-memory load and three dependent operations: one FP64
// instruction of a warp takes 19 cycles of an SM's pipe whatever its active
// lanes and 64 until its result (measured).
//
// One block sweeps one direction for G bands, with three kinds of warps:
//  * one producer copies chunks of SCH positions -- the plan's records, and per
//    band k/D and V Omega/D -- into NCH buffers (cp.async.bulk, completion on
//    an mbarrier), NCH chunks ahead at most;
//  * H helpers turn the chunks' V Omega/D into right-hand sides in place
//    (ebar V Omega/D + boundary part / D, ebar = C_b / Omega_tot (T - T_ref) with
//    T gathered once per block, not ebar per band), and fetch the upstream values that are too old for
//    the ring into the chunk's annex of it;
//  * WC consumer warps per band solve the levels, with a barrier among
//    themselves only: the bands of a block drift apart by up to NCH chunks, so
//    one band's barrier overlaps the others' arithmetic.  A consumer reads
//    records, right-hand sides and upstream values from shared memory alone.
//
// Layout.  A level's positions are ordered by falling inflow count, so that a
// warp can skip the face slots none of its cells has, and padded to rows of 32
// (no cell, zero coefficients): a row is one warp's step without any bounds
// test.  Positions below are padded positions.
// Per cell the arithmetic is k_sweep's in its order, so x is the same to the
// bit.
//
// Measured, one launch in ms by events around it, k_sweep with the shape it is timed
// into -> here: triangles, 1,058 x 5 bands 0.055 -> 0.039, 20,000 x 40 0.529 -> 0.407,
// 25,088 x 20 0.509 -> 0.309, 100,352 x 20 1.50 -> 1.07; tetrahedra, 48,000 x 7
// 1.23 -> 0.89, 131,712 x 20 8.95 -> 6.53.  The FP64 pipe of the SMs with a block is
// 60 to 73 % busy at the large sizes (70 on 100,352 x 20, 73 on 20,000 x 40, 60 on
// 48,000 x 7); a narrow level costs ~500 cycles of control and latency per row.
// Without gain: two bands per consumer warp, unpadded rows, every helper on
// every chunk.
#pragma once
#include "bte_transport.cuh"

namespace bte {

constexpr int SCH = 128;       // positions per chunk
constexpr int SNCH_MAX = 16;   // chunk buffers at most (a power of two)
constexpr int STHREADS = 768;   // threads per block at most (80 registers)

// A chunk's records, by array: int4 (cell or -1, its boundary row + 1 or 0 with
// bit 28 + f set when some cell of the row of 32 has face slot f >= 1, ring
// offsets in bytes of face slots 0 and 1), for FM > 2 int2 (slots 2 and 3),
// then double2 (coefficients 0 and 1) and double / double2 (2 / 2 and 3): loads
// of 8 or 16 bytes per lane without bank conflicts.
template <int FM>
struct StreamRec {
    static constexpr int more = 16, cf = FM > 2 ? 24 : 16, cf2 = cf + 16;  // byte offsets / position
    static constexpr int bytes = FM == 2 ? 32 : FM == 3 ? 48 : 56;         // per position
};

// Where an upstream value is read.  The ring keeps the last W solved positions
// of a band (position p at p mod W), then one place that stays zero (no
// upstream cell), then NCH annexes of A places, one per chunk buffer.
struct StreamShape {
    int G, WC, H; // bands per block, consumer warps per band, helper warps
    int W, A;     // ring positions (a power of two), annex places per chunk
    int NCH;      // chunk buffers (a power of two)
    int cap;      // positions of the widest level
};
__host__ __device__ constexpr int stream_ring(int W, int A, int NCH) { return W + 2 + NCH * ((A + 1) / 2 * 2); }
// Bytes per position of the buffers: its record, and per band k/D and V Omega/D.
template <int FM>
__host__ __device__ constexpr size_t stream_position_bytes(int G) { return StreamRec<FM>::bytes + 16 * (size_t)G; }
constexpr int kStreamHeader = 3 * SNCH_MAX * 8 + 16;
template <int FM>
__host__ __device__ constexpr size_t stream_smem_bytes(const StreamShape& s) {
    return kStreamHeader + sizeof(double) * (size_t)s.G * stream_ring(s.W, s.A, s.NCH) +
           (size_t)s.NCH * SCH * stream_position_bytes<FM>(s.G);
}
// Positions at most `near` back (near = W - cap) are still in the ring
// throughout the level that reads them; older ones come from the annex.  They
// have been written when the helpers fetch them, NCH chunks ahead of their use
// at most, if W >= cap + (NCH + 1) SCH.  A consumer loads a row of 32 positions
// before it releases the chunk of its row before, at most 2 WC x 32 - 32
// positions apart (rows of one level, or the last of one and the first of the
// next): both must fit in the NCH buffers.  A barrier's parity tells
// two successive phases apart only, so whoever waits for a chunk must have seen
// the chunk before it in the same buffer: a helper has if H divides NCH.
__host__ __device__ constexpr int stream_cap(int W, int NCH) { return W - (NCH + 1) * SCH; }  // (a multiple of 32)
__host__ __device__ constexpr bool stream_shape_ok(const StreamShape& s) {
    return s.NCH >= 4 && s.NCH <= SNCH_MAX && (s.NCH & (s.NCH - 1)) == 0 && s.H >= 1 && s.NCH % s.H == 0 && s.cap >= 32 && s.cap <= stream_cap(s.W, s.NCH) &&
           (2 * s.WC * 32 + 126) / SCH <= s.NCH - 1 && s.G <= 15;
}

// Padded position of every cell, spos[d][cell], and its inverse cell[d][pos]
// (-1 where none: set before), from the cell-index order lo_perm of the levels:
// level l of direction d starts at row lvl_row[lvl_off[d] + l].  One warp per
// level; lvl, lvl_off as in SweepPlan.
__global__ void k_stream_order(const int* __restrict__ lo_perm, const uint8_t* __restrict__ mask,
                               const int* __restrict__ lvl, const int* __restrict__ lvl_off,
                               const int* __restrict__ lvl_row, int n, int F, size_t npad, int* __restrict__ spos,
                               int* __restrict__ cell) {
    const int d = blockIdx.y;
    const int lane = threadIdx.x & 31;
    const int l = lvl_off[d] + (int)((blockIdx.x * blockDim.x + threadIdx.x) >> 5);
    if (l + 1 >= lvl_off[d + 1]) return;
    const int* src = lo_perm + (size_t)d * n;
    const uint8_t* md = mask + (size_t)d * n;
    const int j0 = lvl[l], j1 = lvl[l + 1];
    int out = 32 * lvl_row[l];
    for (int k = F; k >= 0; --k)
        for (int j = j0; j < j1; j += 32) {
            const int c = j + lane < j1 ? src[j + lane] : -1;
            const bool take = c >= 0 && __popc((unsigned)md[max(c, 0)]) == k;
            const unsigned m = __ballot_sync(0xffffffffu, take);
            if (take) {
                const int p = out + __popc(m & ((1u << lane) - 1u));
                spos[(size_t)d * n + c] = p;
                cell[(size_t)d * npad + p] = c;
            }
            out += __popc(m);
        }
}

// The diagonal folded into the sweep's coefficients per band and padded
// position, as k_sweep_invd: voi = vo / D, kinv = k_b / D (0
// where there is no cell).
__global__ void k_stream_invd(const int* __restrict__ cell, const double* __restrict__ dg,
                              const double* __restrict__ vo, const double* __restrict__ kb, int n_band, int n_dir,
                              size_t Np, size_t npad, double* __restrict__ voi, double* __restrict__ kinv) {
    const size_t p = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    const int d = blockIdx.y;
    if (p >= npad) return;
    const int c = cell[(size_t)d * npad + p];
    const double g = c >= 0 ? dg[(size_t)d * Np + c] : 0.0, v = c >= 0 ? vo[(size_t)d * Np + c] : 0.0;
    for (int b = 0; b < n_band; ++b) {
        const size_t q = ((size_t)b * n_dir + d) * npad + p;
        const double invD = c >= 0 ? 1.0 / fma(kb[b], g, v) : 0.0;
        voi[q] = v * invD;
        kinv[q] = kb[b] * invD;
    }
}

struct StreamBuild {
    const int* cell;    // [n_dir][npad]
    const int* spos;    // [n_dir][n]
    const int* bidx;    // [n] boundary row of a cell or -1
    const int* nbr;     // [n][F]
    const double* fc;   // [n_dir][F][Np]
    const int* lagged;  // [n_dir][F][n] 0/1, or null: none
    int n, F, nq;       // cells, faces, chunks per direction
    size_t Np, npad;
};

// Upstream values of a chunk that its annex must hold: lagged ones and those
// more than near positions back.  One warp per (direction, chunk).
// BUILD = false: the largest count into *most.  BUILD = true: the records, and
// the annex entries far[(d nq + q) FM SCH ..] (the cell; bit 30 set: lagged)
// with their count in nfar[d nq + q].  Face slots are k_sweep_layout's: inflow
// faces first, in face order.
template <int FM, bool BUILD>
__global__ void k_stream_records(StreamBuild sb, StreamShape sh, int near, unsigned char* __restrict__ rec,
                                 unsigned* __restrict__ far, int* __restrict__ nfar, int* __restrict__ most) {
    using L = StreamRec<FM>;
    const int d = blockIdx.y;
    const int lane = threadIdx.x & 31;
    const int q = (int)((blockIdx.x * blockDim.x + threadIdx.x) >> 5);
    if (q >= sb.nq) return;
    const int annex = sh.W + 2 + (q & (sh.NCH - 1)) * ((sh.A + 1) / 2 * 2);
    int count = 0;
    for (int r = 0; r < SCH / 32; ++r) {
        const int p = q * SCH + r * 32 + lane;
        const int c = sb.cell[(size_t)d * sb.npad + p];
        int u[FM];
        unsigned from[FM];
        double cf[FM];
#pragma unroll
        for (int k = 0; k < FM; ++k) {
            u[k] = -1;
            from[k] = 0;
            cf[k] = 0.0;
        }
        if (c >= 0) {
            int k = 0;
            for (int f = 0; f < sb.F; ++f) {
                const double v = sb.fc[((size_t)d * sb.F + f) * sb.Np + c];
                if (v == 0.0) continue;
                const int o = sb.nbr[(size_t)c * sb.F + f];
                const bool lag = sb.lagged && sb.lagged[((size_t)d * sb.F + f) * sb.n + c];
#pragma unroll
                for (int m = 0; m < FM; ++m)
                    if (m == k) {
                        cf[m] = v;
                        u[m] = lag ? -2 : sb.spos[(size_t)d * sb.n + o];
                        from[m] = (unsigned)o | (lag ? 1u << 30 : 0u);
                    }
                ++k;
            }
        }
        int at[FM];
        unsigned slots = 0;
#pragma unroll
        for (int k = 0; k < FM; ++k) {
            const bool old = u[k] == -2 || (u[k] >= 0 && u[k] < p - near);
            const unsigned m = __ballot_sync(0xffffffffu, old);
            const int a = count + __popc(m & ((1u << lane) - 1u));
            count += __popc(m);
            if (k > 0 && __any_sync(0xffffffffu, u[k] != -1)) slots |= 1u << (28 + k);
            at[k] = 8 * (u[k] == -1 ? sh.W : old ? annex + a : (u[k] & (sh.W - 1)));
            if (BUILD && old) far[((size_t)d * sb.nq + q) * (FM * SCH) + a] = from[k];
        }
        if (BUILD) {
            unsigned char* R = rec + ((size_t)d * sb.npad + (size_t)q * SCH) * L::bytes;
            const int l = r * 32 + lane;
            reinterpret_cast<int4*>(R)[l] = make_int4(c, (int)((unsigned)(c >= 0 ? sb.bidx[c] + 1 : 0) | slots), at[0], at[1]);
            reinterpret_cast<double2*>(R + L::cf * SCH)[l] = make_double2(cf[0], cf[1]);
            if constexpr (FM > 2) {
                reinterpret_cast<int2*>(R + L::more * SCH)[l] = make_int2(at[2], FM > 3 ? at[FM - 1] : 8 * sh.W);
                if constexpr (FM == 3) reinterpret_cast<double*>(R + L::cf2 * SCH)[l] = cf[2];
                else reinterpret_cast<double2*>(R + L::cf2 * SCH)[l] = make_double2(cf[2], cf[3]);
            }
        }
    }
    if (lane == 0) {
        if (BUILD) nfar[(size_t)d * sb.nq + q] = count;
        else if (count > 0) atomicMax(most, count);
    }
}

struct StreamPlan {
    const unsigned char* rec;  // [n_dir][npad]
    const unsigned* far;       // [n_dir][nq][FM SCH]
    const int* nfar;           // [n_dir][nq]
    const int* lrow;           // per direction: start rows of its levels, then its rows
    const int* lvl_off;        // [n_dir + 1]
    int nq;                    // chunks of the longest direction: npad = nq SCH
};

// One wait for the phase of the given parity, for as long as the hardware
// suspends a thread (no time hint: with one the wait becomes a polling loop).
__device__ __forceinline__ bool mbar_try_wait_hw(unsigned long long* bar, unsigned parity) {
    unsigned ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(smem_addr(bar)), "r"(parity)
        : "memory");
    return ok != 0;
}
__device__ __forceinline__ unsigned long long global_ns() {
    unsigned long long t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}
constexpr unsigned long long kStreamWaitNs = 2000000000ull;  // a wait gives up after 2 s
__device__ __forceinline__ void mbar_arrive(unsigned long long* bar) {
    asm volatile("mbarrier.arrive.release.cta.shared::cta.b64 _, [%0];" ::"r"(smem_addr(bar)) : "memory");
}
// Barrier among the nt threads that use named barrier id.
__device__ __forceinline__ void named_barrier(int id, int nt) {
    asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(nt) : "memory");
}

// Grid (ceil(nbb / G), n_dir); (G WC + H + 1) warps.  x = e_curr, x_old =
// e_prev ([band][n_dir][Np]); kinv, voi [band][n_dir][npad] (all bands).  A wait
// that runs out (kStreamWaitNs) sets *err and the block's dead
// flag: every later wait of the block then returns at once, no position is
// solved any more, the barriers are still passed, and the block ends (x is not
// valid; the host reports the error).
template <int FM>
__global__ void __launch_bounds__(STHREADS, 1) k_sweep_stream(StreamPlan sp, StreamShape sh,
                                                          const double* __restrict__ kinv,
                                                          const double* __restrict__ voi, SweepSrc src, double* x,
                                                          int first_sweep, int nbb, int b0, int n_dir, size_t Np,
                                                          int* err) {
    using L = StreamRec<FM>;
    extern __shared__ __align__(128) unsigned char smem[];
    unsigned long long* full = reinterpret_cast<unsigned long long*>(smem);  // [NCH] copies landed
    unsigned long long* ready = full + SNCH_MAX;                             // [NCH] right-hand sides formed
    unsigned long long* empty = ready + SNCH_MAX;                            // [NCH] chunk solved by every consumer
    volatile int* dead = reinterpret_cast<volatile int*>(empty + SNCH_MAX);
    const int ring_len = stream_ring(sh.W, sh.A, sh.NCH);
    double* ring = reinterpret_cast<double*>(smem + kStreamHeader);          // [G][ring_len]
    // NCH chunks of positions, position j at j mod (NCH SCH): records, then per
    // band k/D and V Omega/D (later the right-hand sides)
    const int span = sh.NCH * SCH;
    unsigned char* recs = smem + kStreamHeader + sizeof(double) * (size_t)sh.G * ring_len;
    double* vals = reinterpret_cast<double*>(recs + (size_t)span * L::bytes);  // [G][2][span]
    const int d = blockIdx.y;
    const int g0 = blockIdx.x * sh.G;
    const int gn = min(sh.G, nbb - g0);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const size_t npad = (size_t)sp.nq * SCH;
    const int* lv = sp.lrow + sp.lvl_off[d];
    const int ns = sp.lvl_off[d + 1] - sp.lvl_off[d] - 1;
    const int rows = lv[ns], nq = (rows + SCH / 32 - 1) / (SCH / 32);
    const int qmask = sh.NCH - 1, qshift = __ffs(sh.NCH) - 1;
    if (threadIdx.x == 0) {
        *dead = 0;
        for (int q = 0; q < sh.NCH; ++q) {
            mbar_init(&full[q], 1);
            mbar_init(&ready[q], 1);
            mbar_init(&empty[q], (unsigned)(gn * sh.WC));
        }
        mbar_init_fence();
    }
    if ((int)threadIdx.x < gn) ring[(size_t)threadIdx.x * ring_len + sh.W] = 0.0;
    __syncthreads();
    auto wait = [&](unsigned long long* bar, unsigned parity) -> bool {
        if (mbar_try_wait_hw(bar, parity)) return true;
        const unsigned long long t0 = global_ns();
        for (;;) {
            if (mbar_try_wait_hw(bar, parity)) return true;
            if (*dead) return false;
            if (global_ns() - t0 > kStreamWaitNs) break;
        }
        *dead = 1;
        atomicExch(err, 1);
        return false;
    };

    const int nc = sh.G * sh.WC;  // consumer warps
    if (warp == nc + sh.H) {  // ---- producer
        if (lane != 0) return;
        const unsigned char* rec_d = sp.rec + (size_t)d * npad * L::bytes;
        bool ok = true;
        int q = 0;
        for (; q < nq; ++q) {
            const int slot = q & qmask;
            if (q >= sh.NCH) {
                ok = wait(&empty[slot], (unsigned)((q >> qshift) - 1) & 1u);
                if (!ok) break;
                fence_proxy_async_smem();  // the block's accesses to the buffer come before the copies into it
            }
            const int j = q * SCH;
            constexpr unsigned rb = SCH * (unsigned)L::bytes, vb = SCH * 8u;
            mbar_arrive_expect_tx(&full[slot], rb + 2u * (unsigned)gn * vb);
            bulk_load(recs + (size_t)slot * SCH * L::bytes, rec_d + (size_t)j * L::bytes, rb, &full[slot]);
            double* to = vals + slot * SCH;
            for (int g = 0; g < gn; ++g) {
                const size_t row = ((size_t)(b0 + g0 + g) * n_dir + d) * npad + j;
                bulk_load(to + (size_t)(2 * g) * span, kinv + row, vb, &full[slot]);
                bulk_load(to + (size_t)(2 * g + 1) * span, voi + row, vb, &full[slot]);
            }
        }
        // copies still in flight land in this block's shared memory: it must not end before them
        const unsigned long long t0 = global_ns();
        for (int p = max(0, q - sh.NCH); p < q; ++p)
            while (!mbar_try_wait_hw(&full[p & qmask], (unsigned)(p >> qshift) & 1u) && global_ns() - t0 < kStreamWaitNs) {
            }
        return;
    }

    if (warp >= nc) {  // ---- helpers
        // Helper h takes chunks h, h + H, ...: a chunk is a chain of global
        // loads (entries of the plan, then values), so the helpers work on
        // different chunks at once, and the entries of the next are loaded
        // while this one is worked on.
        const int h = warp - nc;
        const int* nf = sp.nfar + (size_t)d * sp.nq;
        const unsigned* fd = sp.far + (size_t)d * sp.nq * (FM * SCH);
        const size_t row = ((size_t)(b0 + g0) * n_dir + d) * Np, band = (size_t)n_dir * Np;
        constexpr int R = SCH / 32;
        const double cs = lane < gn ? src.Cb[b0 + g0 + lane] / src.solid_angle : 0.0;  // band g's in lane g
        int m = h < nq ? nf[h] : 0, m2 = h + sh.H < nq ? nf[h + sh.H] : 0;
        unsigned e[R];
#pragma unroll
        for (int r = 0; r < R; ++r) e[r] = r * 32 + lane < m ? fd[(size_t)h * (FM * SCH) + r * 32 + lane] : 0u;
        for (int q = h; q < nq; q += sh.H) {
            const int slot = q & qmask;
            if (!wait(&full[slot], (unsigned)(q >> qshift) & 1u)) return;
            const unsigned char* B = recs + (size_t)slot * SCH * L::bytes;
            int bi[R];
            double T[R];
            bool wall = false;
#pragma unroll
            for (int r = 0; r < R; ++r) {
                const int l = r * 32 + lane;
                const int2 cb = *reinterpret_cast<const int2*>(B + l * 16);
                T[r] = cb.x >= 0 ? src.T[cb.x] : 0.0;
                bi[r] = (cb.y & 0x0fffffff) - 1;
                wall |= bi[r] >= 0;
            }
            // old upstream values: the chunk's annex of every band's ring
            double* annex = ring + sh.W + 2 + slot * ((sh.A + 1) / 2 * 2) + lane;
            for (int a = 0; a < m; a += SCH) {
                const unsigned* fe = fd + (size_t)q * (FM * SCH) + a + lane;
                for (int g = 0; g < gn; ++g) {
                    double v[R];
#pragma unroll
                    for (int r = 0; r < R; ++r) {
                        if (a + r * 32 + lane >= m) continue;
                        const unsigned ea = a == 0 ? e[r] : fe[r * 32];
                        v[r] = ((ea >> 30) && first_sweep ? src.x_old : x)[row + g * band + (ea & 0x3fffffffu)];
                    }
#pragma unroll
                    for (int r = 0; r < R; ++r)
                        if (a + r * 32 + lane < m) annex[(size_t)g * ring_len + a + r * 32] = v[r];
                }
            }
            m = m2;
            const int qn = q + sh.H;
            m2 = qn + sh.H < nq ? nf[qn + sh.H] : 0;
#pragma unroll
            for (int r = 0; r < R; ++r) e[r] = r * 32 + lane < m ? fd[(size_t)qn * (FM * SCH) + r * 32 + lane] : 0u;
            wall = __any_sync(0xffffffffu, wall);
            // right-hand sides
            double* kv = vals + slot * SCH + lane;
#pragma unroll
            for (int r = 0; r < R; ++r) T[r] -= src.T_ref;
            for (int g = 0; g < gn; ++g) {
                const double cg = __shfl_sync(0xffffffffu, cs, g);
                double bs[R] = {};
                if (wall) {
                    const double* bb = src.bsum + ((size_t)d * nbb + g0 + g) * src.nbcell;
#pragma unroll
                    for (int r = 0; r < R; ++r)
                        if (bi[r] >= 0) bs[r] = bb[bi[r]];
                }
#pragma unroll
                for (int r = 0; r < R; ++r) {
                    double* v = kv + (size_t)(2 * g + 1) * span + r * 32;
                    *v = fma(cg * T[r], *v, bs[r]);
                }
            }
            fence_proxy_async_smem();
            __syncwarp();
            if (lane == 0) mbar_arrive(&ready[slot]);
        }
        return;
    }

    // ---- consumers: WC warps of band g
    const int g = warp / sh.WC, wl = warp - g * sh.WC;
    if (g >= gn) return;
    double* xb = x + ((size_t)(b0 + g0 + g) * n_dir + d) * Np;
    unsigned char* rg = reinterpret_cast<unsigned char*>(ring + (size_t)g * ring_len);
    const int wmask = sh.W - 1, pmask = span - 1, WC = sh.WC;
    const double* kd = vals + (size_t)(2 * g) * span;  // k/D, then right-hand sides
    constexpr int RCH = SCH / 32;  // rows per chunk
    int known = 0;  // rows (whole chunks) known to be ready
    int done = 0;   // rows (whole chunks) released
    bool ok = true;
    // row r is in its buffer, right-hand sides formed
    auto need = [&](int r) {
        for (; known <= r; known += RCH) {
            const int slot = (known / RCH) & qmask;
            const unsigned parity = (unsigned)((known / RCH) >> qshift) & 1u;
            if (ok) ok = wait(&ready[slot], parity) && wait(&full[slot], parity);
        }
    };
    // chunks before row `upto` are done with.  A chunk is released only once it
    // has been seen ready, lest the arrival count for the chunk before it in the
    // same buffer.
    auto release = [&](int upto) {
        if (done + RCH > upto) return;
        __syncwarp();  // every lane's reads of the chunks and stores of x come before the release
        for (; done + RCH <= upto; done += RCH)
            if (lane == 0) mbar_arrive(&empty[(done / RCH) & qmask]);
    };
    struct Item {
        int c, u[FM];
        double cf[FM], kinv, rhs;
        unsigned slots;  // bit 28 + f: some cell of the row has face slot f >= 1
    };
    auto load = [&](int r, Item& it) {
        const int p = (32 * r + lane) & pmask, l = p & (SCH - 1);
        const unsigned char* R = recs + (p - l) * L::bytes;
        const int4 v = reinterpret_cast<const int4*>(R)[l];
        const double2 w = reinterpret_cast<const double2*>(R + L::cf * SCH)[l];
        it.c = v.x;
        it.u[0] = v.z;
        it.u[1] = v.w;
        it.cf[0] = w.x;
        it.cf[1] = w.y;
        if constexpr (FM > 2) {
            const int2 v2 = reinterpret_cast<const int2*>(R + L::more * SCH)[l];
            it.u[2] = v2.x;
            if constexpr (FM == 3) it.cf[2] = reinterpret_cast<const double*>(R + L::cf2 * SCH)[l];
            else {
                const double2 w2 = reinterpret_cast<const double2*>(R + L::cf2 * SCH)[l];
                it.u[FM - 1] = v2.y;
                it.cf[2] = w2.x;
                it.cf[FM - 1] = w2.y;
            }
        }
        it.slots = (unsigned)v.y;
        it.kinv = kd[p];
        it.rhs = kd[span + p];
    };
    // level bounds: 32 of them in the warp's registers, the next 32 loaded ahead
    int base = 0, sb = lv[min(lane, ns)], sbn = lv[min(32 + lane, ns)];
    auto bound = [&](int i) {  // i never goes back, nor ahead by more than 1
        if (i - base == 32) {
            base += 32;
            sb = sbn;
            sbn = lv[min(base + 32 + lane, ns)];
        }
        return __shfl_sync(0xffffffffu, sb, i - base);
    };
    // Row by row through a level (rows wl, wl + WC, ... of it), then on to the
    // next level behind the band's barrier.  The row after the current one is
    // loaded before the current one is solved, so a barrier is followed by the
    // loads of upstream values and the FP64 chain only.
    int s = 0;
    int r = wl, rB = bound(min(1, ns)), rC = bound(min(2, ns)), rD = bound(min(3, ns));
    bool has = ns > 0 && r < rB;
    auto step = [&](Item& cur, Item& nxt) {
        const bool last = r + WC >= rB;  // of this level, for this warp
        const int rn = last ? rB + wl : r + WC, re = last ? rC : rB;
        const bool more = rn < re;
        // (a warp without a row in the next level sees this level's to their end)
        const int upto = more ? rn : rB, seen = more ? rn : rB - 1;
        if (seen >= known) need(seen);
        if (more) load(rn, nxt);
        if (has) {
            double off = cur.cf[0] * *reinterpret_cast<const double*>(rg + cur.u[0]);
#pragma unroll
            for (int f = 1; f < FM; ++f)
                if (cur.slots >> (28 + f) & 1u)
                    off = fma(cur.cf[f], *reinterpret_cast<const double*>(rg + cur.u[f]), off);
            const double v = fma(-cur.kinv, off, cur.rhs);
            *reinterpret_cast<double*>(rg + 8 * ((32 * r + lane) & wmask)) = v;
            if (cur.c >= 0) xb[cur.c] = v;
        }
        release(upto);
        if (last) {
            if (WC > 1) named_barrier(1 + g, WC * 32);
            else __syncwarp();
            ++s;
            rB = rC;
            rC = rD;
            rD = bound(min(s + 3, ns));  // (used a level later)
        }
        has = more && ok;  // (after a failed wait nothing is solved any more)
        r = rn;
    };
    Item A, B;
    if (ns > 0) {  // the first row, or the first level's end
        need(min(r, rB - 1));
        if (has) load(r, A);
        release(min(r, rB));
        has = has && ok;
    }
    while (s < ns) {
        step(A, B);
        if (s >= ns) break;
        step(B, A);
    }
}

}  // namespace bte
