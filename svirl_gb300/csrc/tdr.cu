// TDGL time loop with the state on chip: one cooperative launch per call.
//
// The sweeps of td.cu read and write the whole state per launch; for domains up to
// about 10^6 nodes a launch is bound by the latency of a warp's walk down its strip
// and by the launch itself, not by bytes.  Here every CTA keeps one tile of an
// instance in registers and shared memory for the whole call (all time steps):
// psi^(k) of the tile and of a K-node halo, the link factors, the right-hand side and
// the reciprocal diagonal.  A group of K Jacobi sweeps runs inside the tile (sweep l
// is valid l nodes inside the halo's edge, so the halo is recomputed instead of being
// exchanged); every sweep's values stay in shared memory, its rim (what neighbours'
// halos cover) goes to global memory, and the CTAs of the instance meet at a barrier.
// Then each reads its halo (L2) and the residual maxima of the K sweeps, and all decide
// alike whether the loop stops and after which sweep, exactly where a loop of single
// sweeps stops.  Instances of a batch have barriers of their own and advance
// independently.  What bounds it: small domains the barrier (arrival, detection and the
// halo's way through L2, 2.6 us a round), larger tiles the instruction rate (about 42
// per node and sweep, FP64: 20 on a pipe that takes one every 64 cycles).
//
// The arithmetic of a node is that of the sweep kernels (glgpu_td.cuh), so the
// results equal those of the launch-per-sweep loop of td.cu bit for bit.
//
// Reference: svirl/cuda/td.h:4-133 (psi sweep), td.h:310-463 (A sweep),
// svirl/solvers/td.py:157-218,252-325,342-377 (host loops, stop rule).
#include <algorithm>
#include <cmath>
#include <cstring>

#include "glgpu_internal.h"
#include "glgpu_td.cuh"

namespace glgpu {

// Shapes: BX x BY threads, each owning a column of R nodes: a tile of BX x (BY R)
// nodes of which the inner (BX - 2K) x (BY R - 2K) are the CTA's own.  K sweeps of psi
// and KA sweeps of A per round.
template <int BX, int BY, int R, int K, int KA> struct ResShape {
    static constexpr int kBX = BX, kBY = BY, kR = R, kK = K, kKA = KA;
    static constexpr int H = BY * R, IW = BX - 2 * K, IH = H - 2 * K, NT = BX * BY;
    // a CTA's exchange slots hold its rim, the own nodes that lie in a neighbour's halo: two
    // sets of every psi sweep of a round and of the round's last A sweep
    static constexpr bool kAllRim = IW <= 2 * K || IH <= 2 * K;
    static constexpr int SLOT = kAllRim ? IW * IH : IW * IH - (IW - 2 * K) * (IH - 2 * K);
    static constexpr int kSlots = 2 * (K + 1), kRimPer = (SLOT + NT - 1) / NT;
    // place of own node (u, v) in a slot: the K rows at both ends, then the K columns at
    // both sides of the rows between
    __host__ __device__ static constexpr int rim_of(int u, int v) {
        return kAllRim ? v * IW + u
               : v < K ? v * IW + u
               : v >= IH - K ? (K + v - (IH - K)) * IW + u
                             : 2 * K * IW + (v - K) * 2 * K + (u < K ? u : u - (IW - 2 * K));
    }
    // own node at place q
    __host__ __device__ static constexpr int rim_u(int q) {
        return kAllRim || q < 2 * K * IW ? q % IW : ((q - 2 * K * IW) % (2 * K) < K ? (q - 2 * K * IW) % (2 * K) : (q - 2 * K * IW) % (2 * K) + IW - 2 * K);
    }
    __host__ __device__ static constexpr int rim_v(int q) {
        return kAllRim || q < K * IW ? q / IW : (q < 2 * K * IW ? IH - 2 * K + q / IW : K + (q - 2 * K * IW) / (2 * K));
    }
    static_assert(KA <= K && (KA == 1 || KA % 2 == 0), "the halo covers the A sweeps; a round starts with a fresh sweep");
    static_assert(K <= kResSweeps && 4 * R <= 32 && IW >= K && IH >= K, "residual words, link-weight bits, halo within one tile");
};

// One round of the instance's barrier: everything this CTA wrote is visible to the
// CTAs that pass it.  false: the wait ran out (or another CTA's did).  Where instances run
// in waves (`more`), the first barrier of an instance waits for CTAs that may have most of
// another instance's call before them, as long as any call: that wait runs out only when
// nothing has arrived at any instance's barrier during `spins` polls.
__device__ __forceinline__ bool res_barrier(ResGroup* g, unsigned& target, unsigned ncta, LoopState* loop, const ResGroup* groups,
                                            int more, int& s_broken) {
    __syncthreads();
    if (threadIdx.x == 0) {
        const bool patient = more && target == 0u;
        target += ncta;
        __threadfence();
        atomicAdd(&g->arrived, 1u);
        unsigned seen, it = 0, progress = 0;
        const unsigned spins = *(volatile const unsigned*)&loop->spins;
        for (;;) {
            asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(seen) : "l"(&g->arrived) : "memory");
            if ((int)(seen - target) >= 0) break;
            if (++it >= spins || (it & 1023u) == 0u) {
                const bool cut = (*(volatile int*)&loop->err & kErrBarrier) != 0;
                if (!cut) {
                    if (it < spins) continue;
                    unsigned all = 0;
#pragma unroll 1
                    for (int q = patient ? loop->ninst : 0; q-- > 0;) all += *(volatile unsigned*)&groups[q].arrived;
                    if (all != progress) {
                        progress = all;
                        it = 0;
                        continue;
                    }
                }
                atomicOr(&loop->err, kErrBarrier);
                s_broken = 1;
                break;
            }
        }
        __threadfence();
    }
    __syncthreads();
    return s_broken == 0;
}

// Running maximum of |x|, |y| with NaN counted apart (the reference's int conversion
// makes a NaN residual 0).  FP32: one maximum that drops NaN and one that keeps it, as
// three-operand instructions; FP64 on the bit patterns, off the FP64 pipe.
struct ResMaxF {
    float m = 0.f, q = 0.f;
    __device__ __forceinline__ void add(float x, float y) {
        asm("max.abs.f32 %0, %0, %1, %2;" : "+f"(m) : "f"(x), "f"(y));
        asm("max.NaN.abs.f32 %0, %0, %1, %2;" : "+f"(q) : "f"(x), "f"(y));
    }
    __device__ __forceinline__ bool nan() const { return isnan(q); }
    using Bits = unsigned;
    __device__ __forceinline__ Bits bits() const { return __float_as_uint(m); }
    static __device__ __forceinline__ Bits warp_max(Bits b) { return __reduce_max_sync(0xffffffffu, b); }
};
struct ResMaxD {
    unsigned long long m = 0ull;
    bool q = false;
    __device__ __forceinline__ void add1(double x) {
        unsigned long long b = (unsigned long long)__double_as_longlong(x) & 0x7fffffffffffffffull;
        if (b > 0x7ff0000000000000ull) {
            q = true;
            b = 0ull;
        }
        m = b > m ? b : m;
    }
    __device__ __forceinline__ void add(double x, double y) {
        add1(x);
        add1(y);
    }
    __device__ __forceinline__ bool nan() const { return q; }
    using Bits = unsigned long long;
    __device__ __forceinline__ Bits bits() const { return m; }
    static __device__ __forceinline__ Bits warp_max(Bits b) {
        const unsigned hi = (unsigned)(b >> 32);
        const unsigned mh = __reduce_max_sync(0xffffffffu, hi);
        const unsigned ml = __reduce_max_sync(0xffffffffu, hi == mh ? (unsigned)b : 0u);
        return ((unsigned long long)mh << 32) | ml;
    }
};
template <typename T> struct ResMaxOf { using type = ResMaxF; };
template <> struct ResMaxOf<double> { using type = ResMaxD; };

template <typename T, class S> struct ResSmem {
    // psi^(k) .. psi^(k+K) of a round; in the A loop [0] is psi and [1] .. [1 + KA] the
    // iterates (a, b) of the links that start at the nodes.  A ring of zeros around each:
    // the outermost nodes' missing neighbours (their values are not used, only kept finite).
    static constexpr int kBufs = S::kK + 1 > S::kKA + 2 ? S::kK + 1 : S::kKA + 2;
    C2<T> buf[kBufs][S::H + 2][S::kBX + 2];
    int off[S::kR][S::NT];  // a halo node's place in its owner's exchange slot
    // a round's residual maxima as bits: each warp's, the instance's; NaN marks by sweep
    typename ResMaxOf<T>::type::Bits wmax[kResSweeps][32];
    unsigned long long res[kResSweeps];
    int wnan[kResSweeps][32];
    int rnan, broken;
};

template <typename T, class S, int MINB>
__global__ void __launch_bounds__(S::NT, MINB)
k_td_resident(const Inst* __restrict__ insts, const ResTile* __restrict__ tiles, const int* __restrict__ first,
              const int* __restrict__ owner, C2<T>* __restrict__ scratch, ResGroup* __restrict__ groups, LoopState* loop,
              int Nt, int do_psi, int do_A, int more) {
    constexpr int BX = S::kBX, R = S::kR, K = S::kK, KA = S::kKA, H = S::H, NT = S::NT, SLOT = S::SLOT;
    constexpr int RC = R < 4 ? R : 4;  // rows whose updates are in flight together
    constexpr bool kDelta = sizeof(T) == 4;
    using Max = typename ResMaxOf<T>::type;
    extern __shared__ __align__(16) unsigned char s_raw[];
    ResSmem<T, S>& sm = *(ResSmem<T, S>*)s_raw;
    auto& sp = sm.buf;
    const int tid = threadIdx.x, tx = tid % BX, ty = tid / BX, lane = tid & 31, e0 = ty * R;
    const C2<T> z = cmk<T>(T(0), T(0));
    for (int e = tid; e < ResSmem<T, S>::kBufs * (H + 2) * (BX + 2); e += NT) (&sp[0][0][0])[e] = z;
    if (tid == 0) sm.broken = 0;
    __syncthreads();
    // this CTA's exchange slots; another CTA's node is at scratch + off + slot * SLOT
    C2<T>* const mine = scratch + (size_t)blockIdx.x * S::kSlots * SLOT + tid;
    // the rim nodes that this thread stores: their places in a buffer
    int rim[S::kRimPer];
#pragma unroll
    for (int q = 0; q < S::kRimPer; ++q) {
        const int w = tid + q * NT;
        rim[q] = w < SLOT ? (S::rim_v(w) + K + 1) * (BX + 2) + S::rim_u(w) + K + 1 : -1;
    }
    auto store_rim = [&](const C2<T>* buf, C2<T>* out) {
#pragma unroll
        for (int q = 0; q < S::kRimPer; ++q)
            if (rim[q] >= 0) out[q * NT] = buf[rim[q]];
    };

    for (int slot = first[blockIdx.x]; slot < first[blockIdx.x + 1]; ++slot) {
        const ResTile tile = tiles[slot];
        const Inst& I = insts[tile.inst];
        ResGroup* grp = groups + tile.inst;
        const Geo g = I.g;
        const int Nx = g.Nx, Ny = g.Ny;
        const unsigned ncta = (unsigned)tile.ncta;
        unsigned target = 0;
        const bool leader = tile.x0 == 0 && tile.y0 == 0;
        const bool solve_A = do_A && I.solveA;
        const T dt = gsel<T>(I.dt, I.fdt), idx2 = GT(g, idx2), idy2 = GT(g, idy2), idxy = GT(g, idxy);
        uint32_t rt = I.st->rand_t;
        const int i = tile.x0 - K + tx, jb = tile.y0 - K + e0;
        const bool in_x = i >= 0 && i < Nx, own_x = in_x && tx >= K && tx < BX - K;
        // per node of the thread's column, a bit each: in the domain, the CTA's own, updated
        // (it has an x link), start of an x link / a y link; link-weight bits, four each
        unsigned inm = 0u, ownm = 0u, live = 0u, linkx = 0u, linky = 0u, cds = 0u;
        const int node0 = i + Nx * jb;
        auto node = [&](int r) { return node0 + Nx * r; };
        C2<T> p[R], rq[R], ua[R], ub[R], ul[R], ud0 = z;
        T inv[R];
#pragma unroll
        for (int r = 0; r < R; ++r) {
            const int e = e0 + r, j = jb + r;
            const bool in = in_x && j >= 0 && j < Ny;
            p[r] = in ? ((const C2<T>*)I.psi[0])[node(r)] : z;
            rq[r] = ua[r] = ub[r] = ul[r] = z;
            inv[r] = T(0);
            if (in) {
                inm |= 1u << r;
                const unsigned cb = cell_bits(g, I.mt, i, j);
                const unsigned cd = ((GL_MM(cb) || GL_MP(cb)) ? 1u : 0u) | ((GL_PM(cb) || GL_PP(cb)) ? 2u : 0u) |
                                    ((GL_MM(cb) || GL_PM(cb)) ? 4u : 0u) | ((GL_MP(cb) || GL_PP(cb)) ? 8u : 0u);
                cds |= cd << (4 * r);
                if (cd & 3u) live |= 1u << r;
                if (i < Nx - 1) linkx |= 1u << r;
                if (j < Ny - 1) linky |= 1u << r;
                if (own_x && e >= K && e < H - K) {
                    ownm |= 1u << r;
                } else {
                    const int ox = i / S::IW, oy = j / S::IH;
                    sm.off[r][tid] = owner[tile.own0 + oy * tile.ntx + ox] * (S::kSlots * SLOT) +
                                     S::rim_of(i - ox * S::IW, j - oy * S::IH);
                }
            }
        }
        auto bit = [](unsigned m, int r) { return (m >> r & 1u) != 0u; };
        const unsigned halo = inm & ~ownm;

        // link factors of the present A: each CTA tabulates its own nodes' links, and
        // after the barrier reads those around its tile (the FP64 sincos is dear, so no
        // link is computed twice)
        auto refresh_links = [&](const T (&a0)[R], const T (&b0)[R]) -> bool {
            const T sx = dt * idx2, sy = dt * idy2;
            C2<T>* U = (C2<T>*)I.U;
#pragma unroll
            for (int r = 0; r < R; ++r)
                if (bit(ownm, r)) {
                    const unsigned cd = cds >> (4 * r);
                    C2<T> va = z, vb = z;
                    if (bit(linkx, r) && (cd & 2u)) va = cscale(sx, link_U<T>(GT(g, dx) * a0[r]));
                    if (bit(linky, r) && (cd & 8u)) vb = cscale(sy, link_U<T>(GT(g, dy) * b0[r]));
                    U[2 * node(r)] = va;
                    U[2 * node(r) + 1] = vb;
                }
            if (!res_barrier(grp, target, ncta, loop, groups, more, sm.broken)) return false;
            ud0 = z;
#pragma unroll
            for (int r = 0; r < R; ++r) {
                ua[r] = ub[r] = ul[r] = z;  // (all set here: none is kept through the A loop)
                if (bit(inm, r)) {
                    const int n = node(r);
                    ua[r] = __ldcg(&U[2 * n]);
                    ub[r] = __ldcg(&U[2 * n + 1]);
                    if (i > 0) ul[r] = __ldcg(&U[2 * (n - 1)]);
                    if (r == 0 && jb > 0) ud0 = __ldcg(&U[2 * (n - Nx) + 1]);
                }
            }
            return true;
        };
        // A of the links that start at the nodes of `mask`
        auto load_A = [&](T (&a0)[R], T (&b0)[R], unsigned mask) {
            const T* A = (const T*)I.ab[0];
#pragma unroll
            for (int r = 0; r < R; ++r) {
                a0[r] = bit(mask & linkx, r) ? __ldcg(&A[node(r) - (jb + r)]) : T(0);
                b0[r] = bit(mask & linky, r) ? __ldcg(&A[g.Na + node(r)]) : T(0);
            }
        };

        int nan_seen = 0, last_psi = 0, last_A = 0, max_psi = 0, max_A = 0, step = 0;
        long long tot_psi = 0, tot_A = 0;
        int flip = 0, flipA = 0;
        unsigned round = 0;  // residual words of round q are in res[q % 3]
        bool ok = true;
        // sweep l's (0, 1, ...) maximum over this warp's nodes
        auto post_sweep = [&](const Max& mx, bool mine, int l) {
            const auto m = Max::warp_max(mine ? mx.bits() : 0);
            const bool nn = __any_sync(0xffffffffu, mine && mx.nan());
            if (lane == 0) {
                sm.wmax[l][tid >> 5] = m;
                sm.wnan[l][tid >> 5] = nn;
            }
        };
        // the CTA's maxima of a round of nv sweeps into the instance's words, a warp for
        // each sweep (after a __syncthreads; the barrier's first one orders its writes)
        auto post_round = [&](int nv) {
            for (int l = tid >> 5; l < nv; l += NT / 32) {
                const bool have = lane < NT / 32;
                const auto m = Max::warp_max(have ? sm.wmax[l][lane] : 0);
                const bool nn = __any_sync(0xffffffffu, have && sm.wnan[l][lane]);
                if (lane == 0) {
                    atomicMax(&grp->res[round % 3u][l], (unsigned long long)m);
                    if (nn) atomicOr(&grp->nan[round % 3u], 1 << l);
                }
            }
        };
        // after the barrier of a round: its maxima (to be read after the next
        // __syncthreads), and the words of the round after the next are cleared
        auto fetch_round = [&](int nv) {
            if (tid < nv) sm.res[tid] = __ldcg(&grp->res[round % 3u][tid]);
            if (tid == 32 % NT) sm.rnan = __ldcg(&grp->nan[round % 3u]);
            if (leader && tid < kResSweeps) *(volatile unsigned long long*)&grp->res[(round + 2u) % 3u][tid] = 0ull;
            if (leader && tid == 0) *(volatile int*)&grp->nan[(round + 2u) % 3u] = 0;
            ++round;
        };

        if (do_psi) {
            T a0[R], b0[R];
            load_A(a0, b0, ownm);
            ok = refresh_links(a0, b0);
        }
        for (; ok && step < Nt; ++step) {
            if (do_psi) {
                // right-hand side with the Langevin term, reciprocal of the diagonal
                const bool lang = I.lang_psi_on != 0;
                const T lc = gsel<T>(I.lang_psi, I.flang_psi), eps0 = gsel<T>(I.epsilon, I.fepsilon);
                const T* eps_sp = (const T*)I.eps_sp;
#pragma unroll
                for (int r = 0; r < R; ++r) {
                    rq[r] = p[r];
                    inv[r] = T(0);
                    if (bit(inm, r)) {
                        const int n = node(r);
                        if (lang) {
                            rq[r].x = add_noise<T>(rq[r].x, lc, rand_1<T>((uint32_t)n, rt));
                            rq[r].y = add_noise<T>(rq[r].y, lc, rand_2<T>((uint32_t)n, rt));
                        }
                        if (bit(live, r))
                            inv[r] = psi_diag_inv<T>(rq[r], eps_sp ? eps_sp[n] : eps0, cds >> (4 * r) & 15u, dt, idx2, idy2);
                    }
                    sp[0][e0 + r + 1][tx + 1] = p[r];
                }
                __syncthreads();
                int k = 0, stop = 0;
                while (!stop) {
                    // two sets of exchange slots in turn (across time steps too): a set is
                    // written again only after a barrier that its readers have passed
                    C2<T>* const out = mine + (size_t)flip * K * SLOT;
#pragma unroll
                    for (int l = 1; l <= K; ++l) {
                        Max mx;
                        C2<T> below = sp[l - 1][e0][tx + 1];
                        const C2<T> above = sp[l - 1][e0 + R + 1][tx + 1];
                        // per chunk of rows: the x neighbours of all rows first (the compiler
                        // cannot move a shared load above a store of the row before), then the
                        // updates, which do not depend on one another, then the stores
#pragma unroll
                        for (int c = 0; c < R; c += RC) {
                            C2<T> lt[RC], rg[RC], nw[RC];
#pragma unroll
                            for (int q = 0; q < RC; ++q) {
                                lt[q] = sp[l - 1][e0 + c + q + 1][tx];
                                rg[q] = sp[l - 1][e0 + c + q + 1][tx + 2];
                            }
#pragma unroll
                            for (int q = 0; q < RC; ++q) {
                                const int r = c + q, e = e0 + r;
                                // FP64: rows that neither a later sweep nor the result needs (the
                                // tile's first and last) stay off the FP64 pipe
                                nw[q] = p[r];
                                if (sizeof(T) == 4 || ((r >= l || e >= l) && (r < R - l || e < H - l)))
                                    nw[q] = psi_node<T>(lt[q], rg[q], q > 0 ? p[r > 0 ? r - 1 : 0] : below,
                                                        r + 1 < R ? p[r + 1 < R ? r + 1 : r] : above, ul[r], ua[r],
                                                        r > 0 ? ub[r > 0 ? r - 1 : 0] : ud0, ub[r], rq[r], inv[r],
                                                        live >> r & 1u);
                            }
                            below = p[c + RC - 1];
#pragma unroll
                            for (int q = 0; q < RC; ++q) {
                                const int r = c + q;
                                sp[l][e0 + r + 1][tx + 1] = nw[q];
                                // residual of the own rows (nodes outside the domain stay 0)
                                if ((r >= K || e0 + r >= K) && (r < R - K || e0 + r < H - K)) mx.add(nw[q].x - p[r].x, nw[q].y - p[r].y);
                                p[r] = nw[q];
                            }
                        }
                        post_sweep(mx, own_x, l - 1);
                        __syncthreads();
                        store_rim(&sp[l][0][0], out + (l - 1) * SLOT);
                    }
                    post_round(K);
                    if (!(ok = res_barrier(grp, target, ncta, loop, groups, more, sm.broken))) break;
                    fetch_round(K);
                    const C2<T>* const in = scratch + (size_t)flip * K * SLOT;
#pragma unroll
                    for (int r = 0; r < R; ++r) {
                        if (bit(halo, r)) p[r] = __ldcg(in + sm.off[r][tid] + (K - 1) * SLOT);
                        sp[0][e0 + r + 1][tx + 1] = p[r];
                    }
                    __syncthreads();
                    stop = 0;
#pragma unroll
                    for (int l = K; l >= 1; --l)
                        if (sm.res[l - 1] <= I.thr_psi || k + l >= kMaxSweeps) stop = l;
                    const int upto = stop ? stop : K;
                    if (sm.rnan & ((1 << upto) - 1)) nan_seen = 1;
                    if (stop && stop < K) {  // the state is that of an earlier sweep of the round
#pragma unroll
                        for (int r = 0; r < R; ++r)
                            p[r] = bit(halo, r) ? __ldcg(in + sm.off[r][tid] + (stop - 1) * SLOT) : sp[stop][e0 + r + 1][tx + 1];
                    }
                    k += upto;
                    flip ^= 1;
                    __syncthreads();  // the round's words have been read
                }
                if (!ok) break;
                last_psi = k;
                tot_psi += k;
                max_psi = k > max_psi ? k : max_psi;
                rt += 1u;
            }
            if (solve_A) {
                const T k2 = gsel<T>(I.kappa2, I.fkappa2), dt_rho = dt * gsel<T>(I.rho, I.frho), dt_rho_k2 = dt_rho * k2;
                const T Hf = gsel<T>(I.H, I.fH), idx = GT(g, idx), idy = GT(g, idy), dx = GT(g, dx), dy = GT(g, dy);
                const bool lang = I.lang_A_on != 0;
                const T lc = gsel<T>(I.lang_A, I.flang_A);
                const T rh_y = T(2) * k2 * Hf * idy, rh_x = T(2) * k2 * Hf * idx;
                const T den_a = T(1) + T(2) * dt_rho_k2 * idy2, den_b = T(1) + T(2) * dt_rho_k2 * idx2;
                const T rden_a = T(1) / den_a, rden_b = T(1) / den_b;
                // FP32 computes the links of the whole tile (the halo's again in every CTA, KA
                // sweeps per round); FP64 those of the own nodes, a sweep per round (its sincos
                // and divisions are dear)
                const unsigned actm = KA > 1 ? inm : ownm;
                T a0[R], b0[R], ac[R], bc[R], xa[R], xb[R], ga[kDelta ? R : 1], gb[kDelta ? R : 1];
                load_A(a0, b0, inm);
#pragma unroll
                for (int r = 0; r < R; ++r) {
                    sp[0][e0 + r + 1][tx + 1] = p[r];
                    sp[1][e0 + r + 1][tx + 1] = cmk<T>(a0[r], b0[r]);
                    ac[r] = kDelta ? T(0) : a0[r];  // FP32 iterates the offsets from A^(0) (k_A_loop_f32)
                    bc[r] = kDelta ? T(0) : b0[r];
                    xa[r] = xb[r] = T(0);
                }
                __syncthreads();
                // neighbour terms of the node's links from the iterate in sp[c] (the thread's
                // own column from av, bv)
                auto nbs = [&](int c, int r, const T (&av)[R], const T (&bv)[R], T& nx, T& ny) {
                    const int e = e0 + r + 1;
                    const C2<T> dn = r > 0 ? cmk<T>(av[r > 0 ? r - 1 : 0], bv[r > 0 ? r - 1 : 0]) : sp[c][e - 1][tx + 1];
                    const T up = r + 1 < R ? av[r + 1 < R ? r + 1 : r] : sp[c][e + 1][tx + 1].x;
                    const C2<T> lf = sp[c][e][tx];
                    const T rt_b = sp[c][e][tx + 2].y;
                    nx = A_nbs_x<T>(idy2, idxy, dn.x, up, dn.y, sp[c][e - 1][tx + 2].y, bv[r], rt_b);
                    ny = A_nbs_y<T>(idx2, idxy, lf.y, rt_b, lf.x, sp[c][e + 1][tx].x, av[r], up);
                };
                if constexpr (kDelta) {
#pragma unroll
                    for (int r = 0; r < R; ++r) {
                        const int j = jb + r;
                        T nx, ny;
                        nbs(1, r, a0, b0, nx, ny);
                        const T dda = (j == 0 || j == Ny - 1) ? T(2) : T(1), ddb = (i == 0 || i == Nx - 1) ? T(2) : T(1);
                        ga[r] = A_base<T>(dt_rho_k2, dda, nx, idy2, a0[r]);
                        gb[r] = A_base<T>(dt_rho_k2, ddb, ny, idx2, b0[r]);
                    }
                }
                int k = 0, stop = 0;
                while (!stop) {
#pragma unroll
                    for (int l = 1; l <= KA; ++l) {
                        Max mx;
                        const bool fresh = KA > 1 ? (l & 1) == 1 : (k & 1) == 0;
                        const bool zero = kDelta && l == 1 && k == 0;  // the offsets start from zero
                        T va[R], vb[R];
#pragma unroll
                        for (int r = 0; r < R; ++r) {
                            const int e = e0 + r + 1, j = jb + r;
                            va[r] = ac[r];
                            vb[r] = bc[r];
                            if (bit(actm, r)) {
                                const unsigned cd = cds >> (4 * r);
                                const T dda = (j == 0 || j == Ny - 1) ? T(2) : T(1), ddb = (i == 0 || i == Nx - 1) ? T(2) : T(1);
                                if (fresh) {  // the fixed parts, with the supercurrent of A^(k)
                                    const T rha = j == 0 ? rh_y : (j == Ny - 1 ? -rh_y : T(0));
                                    const T rhb = i == 0 ? -rh_x : (i == Nx - 1 ? rh_x : T(0));
                                    const T pha = kDelta ? a0[r] + ac[r] : ac[r], phb = kDelta ? b0[r] + bc[r] : bc[r];
                                    const C2<T> p0 = sp[0][e][tx + 1];
                                    T ja = mul_rn<T>(idx, js_of<T>(p0, dx * pha, sp[0][e][tx + 2]));
                                    T jc = mul_rn<T>(idy, js_of<T>(p0, dy * phb, sp[0][e + 1][tx + 1]));
                                    if (!(cd & 2u)) ja = T(0);
                                    if (!(cd & 8u)) jc = T(0);
                                    const uint32_t na = (uint32_t)(node(r) - j), nb = (uint32_t)(g.Na + node(r));
                                    T fa = kDelta ? T(0) : a0[r], fb = kDelta ? T(0) : b0[r];
                                    if (lang) {
                                        fa = add_noise<T>(fa, lc, rand_1<T>(na, rt));
                                        fb = add_noise<T>(fb, lc, rand_2<T>(nb, rt));
                                    }
                                    xa[r] = A_fixed<T>(fa, dt_rho, ja, rha);
                                    xb[r] = A_fixed<T>(fb, dt_rho, jc, rhb);
                                    if constexpr (kDelta) {
                                        xa[r] += ga[r];
                                        xb[r] += gb[r];
                                    }
                                }
                                T nx = T(0), ny = T(0);
                                if (!zero) nbs(l, r, ac, bc, nx, ny);
                                va[r] = bit(linkx, r) ? div_by(fma(dt_rho_k2 * dda, nx, xa[r]), den_a, rden_a) : T(0);
                                vb[r] = bit(linky, r) ? div_by(fma(dt_rho_k2 * ddb, ny, xb[r]), den_b, rden_b) : T(0);
                            }
                        }
#pragma unroll
                        for (int r = 0; r < R; ++r) {
                            if (bit(ownm, r)) mx.add(va[r] - ac[r], vb[r] - bc[r]);
                            ac[r] = va[r];
                            bc[r] = vb[r];
                            sp[1 + l][e0 + r + 1][tx + 1] = cmk<T>(va[r], vb[r]);
                        }
                        post_sweep(mx, true, l - 1);
                        __syncthreads();
                    }
                    store_rim(&sp[1 + KA][0][0], mine + (2 * K + flipA) * SLOT);
                    post_round(KA);
                    if (!(ok = res_barrier(grp, target, ncta, loop, groups, more, sm.broken))) break;
                    fetch_round(KA);
                    const C2<T>* const in = scratch + (2 * K + flipA) * SLOT;
#pragma unroll
                    for (int r = 0; r < R; ++r) {
                        if (bit(halo, r)) {
                            const C2<T> v = __ldcg(in + sm.off[r][tid]);
                            ac[r] = v.x;
                            bc[r] = v.y;
                        }
                        sp[1][e0 + r + 1][tx + 1] = cmk<T>(ac[r], bc[r]);
                    }
                    __syncthreads();
#pragma unroll
                    for (int l = KA; l >= 1; --l)
                        if (sm.res[l - 1] <= I.thr_A || k + l >= kMaxSweeps) stop = l;
                    const int upto = stop ? stop : KA;
                    if (sm.rnan & ((1 << upto) - 1)) nan_seen = 1;
                    if (stop && stop < KA) {  // (the halo's links are read again with the next step's A)
#pragma unroll
                        for (int r = 0; r < R; ++r) {
                            const C2<T> v = sp[1 + stop][e0 + r + 1][tx + 1];
                            ac[r] = v.x;
                            bc[r] = v.y;
                        }
                    }
                    k += upto;
                    flipA ^= 1;
                    __syncthreads();  // the round's words have been read
                }
                if (!ok) break;
                T* A = (T*)I.ab[0];
#pragma unroll
                for (int r = 0; r < R; ++r) {
                    a0[r] = kDelta ? a0[r] + ac[r] : ac[r];
                    b0[r] = kDelta ? b0[r] + bc[r] : bc[r];
                    if (bit(ownm & linkx, r)) A[node(r) - (jb + r)] = a0[r];
                    if (bit(ownm & linky, r)) A[g.Na + node(r)] = b0[r];
                    p[r] = sp[0][e0 + r + 1][tx + 1];  // (not kept in registers meanwhile)
                }
                last_A = k;
                tot_A += k;
                max_A = k > max_A ? k : max_A;
                rt += 1u;
                // the new A (its factors) before the next step reads it
                if (do_psi) {
                    ok = refresh_links(a0, b0);
                } else {
                    ok = res_barrier(grp, target, ncta, loop, groups, more, sm.broken);
                    ud0 = z;
#pragma unroll
                    for (int r = 0; r < R; ++r) ua[r] = ub[r] = ul[r] = z;
                }
            }
        }
        if (ok && do_psi)
#pragma unroll
            for (int r = 0; r < R; ++r)
                if (bit(ownm, r)) ((C2<T>*)I.psi[0])[node(r)] = p[r];
        if (leader && tid == 0) {
            InstState* st = I.st;
            st->rand_t = rt;
            st->nan_seen = nan_seen;
            st->last_sweeps_psi = last_psi;
            st->last_sweeps_A = last_A;
            st->max_sweeps_psi = max_psi;
            st->max_sweeps_A = max_A;
            st->total_sweeps_psi = tot_psi;
            st->total_sweeps_A = tot_A;
            st->steps = step;
            if (tile.inst == 0) {
                loop->step = step;
                loop->total_launches = 1;
            }
        }
        // a CTA's exchange slots are free for its next instance once all have read them
        if (more && ok) ok = res_barrier(grp, target, ncta, loop, groups, more, sm.broken);
        __syncthreads();
        if (sm.broken) return;
    }
}

// ---------------------------------------------------------------------------
// host side
// ---------------------------------------------------------------------------

struct ResCfg {
    int dtype, nt, iw, ih, nodes, K, smem, most;  // nodes: of a tile, with its halo
    double wave_us;  // a time step of a film among films in waves (0: the shape takes no waves)
    size_t scratch;  // exchange slots of a CTA, bytes
    void* fn;
};
template <typename T, class S, int MINB> static ResCfg res_cfg(int most, double wave_us) {
    return ResCfg{(int)sizeof(T), S::NT, S::IW, S::IH, S::kBX * S::H, S::kK, (int)sizeof(ResSmem<T, S>), most, wave_us,
                  sizeof(C2<T>) * S::kSlots * S::SLOT, (void*)k_td_resident<T, S, MINB>};
}
// Shapes in the order they are tried.  A single FP32 domain takes the first in which it
// has at most `most` tiles (0: as many as CTAs are resident at once), FP64 the one that
// res_sweep_us finds fastest: small tiles with many
// sweeps per round, where the barrier and the halo's way through L2 (2.6 us a round)
// are most of a step, then larger ones.  Batches whose tiles do not all fit run in
// waves on a shape with a wave_us, or in the loops of tdl.cu (res_schedule).  Measured, us
// per time step (22 psi sweeps), by the launch-per-sweep loop and by the shapes here (own
// nodes per tile):
//   FP32, kappa = inf:  129^2 145, 16x16 19;  513^2 164, 58x26 52;  700^2 172, 60x60 72
//   FP32, kappa = 4:    257^2 22x22 39 (16x16 42);  385^2 250, 24x24 53 (58x26 55);
//                       449^2 58x26 56, two CTAs per SM 73
//   FP64, kappa = inf:  129^2 315, 12x12 63 (28x12 93);  257^2 321, 28x12 150 (28x28 162);
//                       385^2 378, 62x14 306 (62x30 323)
//   32 films of 64^2 .. 512^2, 20 steps, FP32: 18.8 ms, in waves of 58x26 tiles 14.0
//   (60x60: 16.0)
static const ResCfg* res_cfgs(int* n) {
    static const ResCfg c[] = {
        res_cfg<float, ResShape<32, 16, 2, 8, 4>, 2>(240, 0.0),   // 16 x 16
        res_cfg<float, ResShape<32, 8, 4, 5, 4>, 2>(0, 0.0),      // 22 x 22
        res_cfg<float, ResShape<32, 8, 4, 4, 4>, 2>(0, 0.0),      // 24 x 24
        res_cfg<float, ResShape<64, 8, 4, 3, 2>, 1>(0, 0.0),      // 58 x 26, a CTA per SM (128 registers)
        res_cfg<float, ResShape<64, 8, 4, 3, 2>, 2>(0, 49.0),     // 58 x 26, two (64 registers, spills)
        res_cfg<float, ResShape<64, 8, 8, 2, 2>, 1>(0, 66.0),     // 60 x 60
        res_cfg<double, ResShape<16, 16, 1, 2, 1>, 2>(230, 0.0),  // 12 x 12
        res_cfg<double, ResShape<32, 8, 2, 2, 1>, 2>(0, 0.0),     // 28 x 12
        res_cfg<double, ResShape<32, 16, 2, 2, 1>, 1>(0, 0.0),    // 28 x 28
        res_cfg<double, ResShape<64, 4, 4, 1, 1>, 2>(0, 0.0),     // 62 x 14
        res_cfg<double, ResShape<64, 8, 4, 1, 1>, 1>(0, 0.0),     // 62 x 30
    };
    *n = (int)(sizeof(c) / sizeof(c[0]));
    return c;
}

// FP64: a sweep's time by a model, us: the FP64 pipe for the tiles of the SM that has the
// most (20 instructions a node, 64 cycles of a scheduler each for 32 nodes) and a barrier
// round for every K sweeps.  It follows the measured times above within 8 %: 257^2 28x12
// 157, 28x28 157; 385^2 62x30 318.  Sizes between the steps: 470 x 230 took 62 x 30 tiles
// on 64 SMs and 323 us per step, 62 x 14 tiles on 136 SMs take 188.
static double res_sweep_us(const ResCfg& c, long long tiles, int sms) {
    return (double)((tiles + sms - 1) / sms) * c.nodes * 0.0052 + 3.6 / c.K;
}

static int res_tiles_of(const ResCfg& c, const Geo& g) {
    return ((g.Nx + c.iw - 1) / c.iw) * ((g.Ny + c.ih - 1) / c.ih);
}

// The schedule of a call over n instances: the shape, and for each CTA of a grid that
// is resident at once its tiles.  Where an instance's A is solved, a step takes about
// 1.8 times as long.  Instances start in one order, the same in every CTA's list, so
// the first unfinished instance always has all its CTAs at work or on the way to it,
// and no barrier waits for a CTA that waits for another.
// Waves or the loops of tdl.cu: a film in a wave takes wave_us a step whatever share of the
// CTAs it uses, so large films (two of 512^2 do not fit together) lose in waves and small ones
// gain, and A costs more there.  us per step, waves / loops: 2 films of 512^2 95 / 166, 4:
// 200 / 207, 8: 375 / 314, 16: 796 / 523; kappa = 4: 171 / 239, 360 / 315, 678 / 473, 1358 /
// 803; 200 of 128^2 482 / 595, kappa = 4 900 / 883; 32 of 65 .. 496, mixed kappa, 520 / 609.
// (0.95: near the line the estimates are as far off, and films in waves do not wait for the
// one with the most sweeps.)
// false: no shape takes the call, or the loops are expected to be faster.
static bool res_schedule(int dtype, glgpu_handle* const* hs, int n, ResPlan* plan) {
    int nc = 0, dev = 0, sms = 0, coop = 0;
    const ResCfg* cs = res_cfgs(&nc);
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, dev);
    if (!coop) return false;
    int best = -1, best_cap = 0;
    double best_us = 0.0;
    bool in_waves = false;
    for (int c = 0; c < nc; ++c) {
        if (cs[c].dtype != dtype) continue;
        int per = 0;
        if (cudaFuncSetAttribute(cs[c].fn, cudaFuncAttributeMaxDynamicSharedMemorySize, cs[c].smem) != cudaSuccess ||
            cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, cs[c].fn, cs[c].nt, (size_t)cs[c].smem) != cudaSuccess)
            continue;
        const int cap = per * sms;
        long long all = 0;
        int largest = 0;
        for (int q = 0; q < n; ++q) {
            const int t = res_tiles_of(cs[c], hs[q]->g);
            all += t;
            largest = std::max(largest, t);
        }
        const bool fits = all <= (cs[c].most > 0 ? std::min(cs[c].most, cap) : cap);
        if (!fits && !(n > 1 && cs[c].wave_us > 0.0 && largest <= cap)) continue;
        const double us = res_sweep_us(cs[c], all, sms);
        if (best >= 0 && us >= best_us) continue;
        best = c;
        best_cap = cap;
        best_us = us;
        in_waves = !fits;
        if (dtype == 4) break;  // in order
    }
    if (best < 0) return false;
    const ResCfg& c = cs[best];
    plan->fn = c.fn;
    plan->threads = c.nt;
    plan->smem = c.smem;
    plan->scratch = c.scratch;
    long long all = 0;
    std::vector<int> left(n), tiles(n);
    for (int q = 0; q < n; ++q) {
        left[q] = q;
        tiles[q] = res_tiles_of(c, hs[q]->g);
        all += tiles[q];
    }
    const int grid = (int)std::min<long long>(all, best_cap);
    // largest first; whenever CTAs get free, the largest instance that fits on the free ones
    std::stable_sort(left.begin(), left.end(), [&](int a, int b) { return tiles[a] > tiles[b]; });
    std::vector<double> busy(grid, 0.0);
    std::vector<std::vector<ResTile>> per(grid);
    std::vector<int> ctas;
    double now = 0.0;
    plan->tiles.clear();
    plan->owner.clear();
    while (!left.empty()) {
        ctas.clear();
        for (int k = 0; k < grid; ++k)
            if (busy[k] <= now) ctas.push_back(k);
        size_t pick = 0;
        while (pick < left.size() && tiles[left[pick]] > (int)ctas.size()) ++pick;
        if (pick == left.size()) {  // none fits: on to the next time that a CTA gets free
            double next = -1.0;
            for (int k = 0; k < grid; ++k)
                if (busy[k] > now && (next < 0.0 || busy[k] < next)) next = busy[k];
            now = next;
            continue;
        }
        const int q = left[pick], nt = tiles[q], nx = (hs[q]->g.Nx + c.iw - 1) / c.iw;
        left.erase(left.begin() + pick);
        for (int t = 0; t < nt; ++t) {
            per[ctas[t]].push_back(ResTile{q, (t % nx) * c.iw, (t / nx) * c.ih, nt, (int)plan->owner.size(), nx});
            busy[ctas[t]] = now + (hs[q]->inst_h.solveA ? 1.8 : 1.0);
        }
        plan->owner.insert(plan->owner.end(), ctas.begin(), ctas.begin() + nt);
    }
    if (in_waves) {
        std::vector<const Geo*> geos(n);
        bool any_A = false;
        for (int q = 0; q < n; ++q) {
            geos[q] = &hs[q]->g;
            any_A = any_A || hs[q]->inst_h.solveA != 0;
        }
        if (loops_step_us(geos.data(), n, any_A) < 0.95 * c.wave_us * *std::max_element(busy.begin(), busy.end())) return false;
    }
    plan->first.assign(1, 0);
    for (int k = 0; k < grid; ++k) {
        plan->tiles.insert(plan->tiles.end(), per[k].begin(), per[k].end());
        plan->first.push_back((int)plan->tiles.size());
    }
    return true;
}

// The schedule, its device copies and the exchange slots, made at the first call of a
// handle or batch (its geometry does not change).  false: the call takes the
// launch-per-sweep loop.
bool res_prepare(ResState* r, glgpu_handle* const* hs, int n) {
    if (r->ready != 0) return r->ready > 0;
    r->ready = -1;
    ResPlan& p = r->plan;
    if (!res_schedule(hs[0]->dtype, hs, n, &p)) return false;
    const size_t tb = sizeof(ResTile) * p.tiles.size(), fb = sizeof(int) * p.first.size(), ob = sizeof(int) * p.owner.size();
    if (cudaMalloc(&r->tiles, tb) != cudaSuccess || cudaMalloc(&r->first, fb) != cudaSuccess ||
        cudaMalloc(&r->owner, ob) != cudaSuccess || cudaMalloc(&r->groups, sizeof(ResGroup) * (size_t)n) != cudaSuccess ||
        cudaMalloc(&r->scratch, p.scratch * (p.first.size() - 1)) != cudaSuccess ||
        cudaMemcpy(r->tiles, p.tiles.data(), tb, cudaMemcpyHostToDevice) != cudaSuccess ||
        cudaMemcpy(r->first, p.first.data(), fb, cudaMemcpyHostToDevice) != cudaSuccess ||
        cudaMemcpy(r->owner, p.owner.data(), ob, cudaMemcpyHostToDevice) != cudaSuccess) {
        cudaGetLastError();
        res_free(r);
        return false;
    }
    r->ready = 1;
    return true;
}

void res_free(ResState* r) {
    void* ptrs[] = {r->tiles, r->first, r->owner, r->groups, r->scratch};
    for (void* q : ptrs)
        if (q) cudaFree(q);
    r->tiles = nullptr;
    r->first = nullptr;
    r->owner = nullptr;
    r->groups = nullptr;
    r->scratch = nullptr;
}

cudaError_t res_launch(const ResState& r, const Inst* insts, int ninst, LoopState* loop, int Nt, int eqn, cudaStream_t s) {
    int do_psi = eqn != 2, do_A = eqn != 1, more = ninst > 1 ? 1 : 0;
    const ResTile* tiles = r.tiles;
    const int *first = r.first, *owner = r.owner;
    void* scratch = r.scratch;
    ResGroup* groups = r.groups;
    void* a[] = {&insts, &tiles, &first, &owner, &scratch, &groups, &loop, &Nt, &do_psi, &do_A, &more};
    return cudaLaunchCooperativeKernel(r.plan.fn, dim3((unsigned)r.plan.first.size() - 1u), dim3(r.plan.threads), a,
                                       (size_t)r.plan.smem, s);
}

// The largest residual that meets the stop rule (jacobi_converged, monotone in the
// residual), as IEEE bits, so that the device loop compares integers
// (the rule's FP64 division takes the GPU about a microsecond).
unsigned long long res_threshold(int dtype, double stop) {
    // (int)x < 10000 in the rule; a NaN x (an infinite residual against an infinite
    // criterion) becomes 0 there
    auto conv = [&](unsigned long long b) {
        if (dtype == 4) {
            float r;
            const uint32_t u = (uint32_t)b;
            memcpy(&r, &u, 4);
            return !((float)((1.0e4 * (double)r) / (double)(float)stop) >= 10000.0f);
        }
        double r;
        memcpy(&r, &b, 8);
        return !((1.0e4 * r) / stop >= 10000.0);
    };
    unsigned long long lo = 0, hi = dtype == 4 ? 0x7f800000ull : 0x7ff0000000000000ull;  // conv(0)
    if (conv(hi)) return hi;
    while (hi - lo > 1) {
        const unsigned long long m = lo + (hi - lo) / 2;
        if (conv(m)) lo = m;
        else hi = m;
    }
    return lo;
}

}  // namespace glgpu
