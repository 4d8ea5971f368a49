// The Jacobi loop of the psi step as one cooperative launch, for the domains and calls
// that the resident time loop (tdr.cu) does not take: the state stays in global memory,
// the CTAs work through tiles of every instance in rounds of one (FP64) or three (FP32)
// sweeps, and the CTA that finishes a round last decides which instances go on.  A launch
// per round inside a conditional graph node costs about 8 us more than a round here.
// Node arithmetic: glgpu_td.cuh, so states and sweep counts equal those of single sweeps.
//
// Reference: svirl/cuda/td.h:4-133 (psi sweep), svirl/solvers/td.py:157-218 (host loop,
// stop rule).
#include <algorithm>
#include <cmath>
#include <type_traits>

#include "glgpu_bulk.cuh"
#include "glgpu_internal.h"
#include "glgpu_td.cuh"

namespace glgpu {

// Buffer of psi^(s), s a multiple of the sweeps per round and round = s / K the number of
// finished rounds: psi^(0), the right-hand side, stays in R and the two after it take turns.
__device__ __forceinline__ int ring_of(int R, int round) { return round == 0 ? R : (R + 1 + (round - 1) % 2) % kPsiBufs; }
// Buffer of sweep l < K of a round, where it is kept (FP32).
__device__ __forceinline__ int mid_of(int R, int l) { return (R + 2 + l) % kPsiBufs; }

// End of a round: the CTA that arrives last closes it for every instance whose loop still
// runs (close(instance, state): bit 0 the loop goes on, bit 1 it has reached the guard),
// decides whether one is left, and publishes round and decision in one word.  What the CTAs
// wrote in the round is visible after it.  false: leave the loop (finished, or a wait ran
// out).  The word of a round stays until this CTA has arrived at the next one, so nobody
// misses it.
template <typename Close>
__device__ __forceinline__ bool end_round(const Inst* insts, int ninst, LoopState* loop, int seq, int& s_word, const Close& close) {
    __syncthreads();
    if (threadIdx.x == 0) {
        __threadfence();
        s_word = atomicAdd(&loop->arrived, 1u) + 1u == (unsigned)seq * gridDim.x ? -1 : 0;
    }
    __syncthreads();
    if (s_word < 0) {
        int flags = 0;
        __threadfence();
        for (int q = threadIdx.x; q < ninst; q += blockDim.x) {
            InstState* st = insts[q].st;
            if (*(volatile const int*)&st->done) continue;
            flags |= close(insts[q], st);
            __threadfence();
        }
        int left = __syncthreads_or(flags & 1);
        const int cut = __syncthreads_or(flags & 2);
        if (threadIdx.x == 0) {
            if (seq == 1) loop->total_launches += 1;
            if (!left) loop->active = 0;
            if (left && cut) {
                left = 0;
                loop->err |= kErrLoopGuard;
            }
            left = left ? 1 : 0;
            loop->cont = left;
            s_word = 2 * seq + left;
            __threadfence();
            asm volatile("st.release.gpu.global.u32 [%0], %1;" ::"l"(&loop->round), "r"(s_word) : "memory");
        }
    } else if (threadIdx.x == 0) {
        unsigned word, it = 0;
        const unsigned spins = *(volatile const unsigned*)&loop->spins;
        for (;;) {
            asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(word) : "l"(&loop->round) : "memory");
            if (word >> 1 == (unsigned)seq) break;
            if (++it >= spins || ((it & 1023u) == 0u && (*(volatile int*)&loop->err & kErrBarrier))) {
                atomicOr(&loop->err, kErrBarrier);
                word = 0u;
                break;
            }
        }
        __threadfence();
        s_word = (int)word;
    }
    __syncthreads();
    return s_word & 1;
}

// The residual words of an instance's round, read and cleared; the first of its sweeps k + 1
// .. k + K that meets the stop rule or the sweep cap (0: none), not past `guard` sweeps.
template <int K>
__device__ __forceinline__ int stop_level(InstState* st, int k, unsigned long long thr, int guard) {
    unsigned long long res[K];
#pragma unroll
    for (int l = 0; l < K; ++l) res[l] = atomicExch(&st->resp[l], 0ull);
    const int nl = atomicExch(&st->nanlv, 0);
    int stop = 0;
#pragma unroll
    for (int l = K; l >= 1; --l)
        if ((res[l - 1] <= thr || k + l >= kMaxSweeps) && k + l <= guard) stop = l;
    if (nl & ((1 << (stop ? stop : K)) - 1)) st->nan_seen = 1;
    return stop;
}

// Closes a psi round of K sweeps.  An instance whose loop stops after a sweep that the round
// did not keep repeats it up to there in the next round (InstState::redo).
template <int K> struct ClosePsi {
    int round, first, guard;  // guard in sweeps
    __device__ __forceinline__ int operator()(const Inst& I, InstState* st) const {
        const int R = *(volatile const int*)&st->rhs, redo = *(volatile const int*)&st->redo;
        const int k = K * (round - (redo ? 1 : 0)), base = K * first;
        int stop = redo ? redo : stop_level<K>(st, k, I.thr_psi, guard + base);
        if (first > 0) stop = 0;  // a timed loop runs for `guard` sweeps whatever they find
        if (!stop || (!redo && stop < K && !*(volatile const int*)&st->keep)) {
            st->redo = stop;
            // the next round keeps every sweep if the step before stopped within it
            const int ls = *(volatile const int*)&st->last_sweeps_psi;
            st->keep = !stop && K > 1 && (ls == 0 || (ls > k + K && ls < k + 2 * K));
            return 1 | (!stop && k + K >= guard + base ? 2 : 0);
        }
        const int s = k + stop;
        st->sweep = s;
        st->done = 1;
        st->redo = 0;
        st->rhs = stop == K ? ring_of(R, k / K + 1) : mid_of(R, stop);
        st->last_sweeps_psi = s;
        st->total_sweeps_psi += s;
        if (s > st->max_sweeps_psi) st->max_sweeps_psi = s;
        return 0;
    }
};

// FP64: one sweep per round, a node per thread.  The FP64 pipe bounds it (20 FP64
// instructions a node; a warp instruction takes 64 cycles of its scheduler), so nothing
// is recomputed: fused sweeps in strips of 32 x 17 nodes spent 1.4 times the
// instructions.  The five psi values and the link factors of a node come from L1/L2,
// which are far from their limits.  A CTA's threads stride over the tiles (256
// consecutive nodes).  All instances are at the same sweep of their loops, so a round's
// buffers follow from its number, and of the loop state only `done` is read again.
// Only whether a residual meets the stop rule counts, so where a CTA already holds one
// that does not, the differences (two of the FP64 instructions) are left out.
// Sweep at 1025 x 1025: 43 us, 38 of them FP64 pipe (46 with the descriptor and the tile
// table read again from L2 in every round), against 72 for a third of a strip
// launch of three sweeps inside a conditional graph node (513^2: 18.8 against 23, 65^2: 7.4
// against 15; as a launch per sweep in the conditional node 61, 26 and 14).
__device__ __forceinline__ void flush_f64(const Inst& I, unsigned long long rmax, bool nan, unsigned long long* s_max) {
    const int lane = threadIdx.x & 31;
    const unsigned hi = __reduce_max_sync(0xffffffffu, (unsigned)(rmax >> 32));
    const unsigned lo = __reduce_max_sync(0xffffffffu, (unsigned)(rmax >> 32) == hi ? (unsigned)rmax : 0u);
    const bool any_nan = __any_sync(0xffffffffu, nan);
    if (lane == 0) {
        s_max[threadIdx.x >> 5] = (unsigned long long)hi << 32 | lo;
        if (any_nan) atomicOr(&I.st->nanlv, 1);
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        unsigned long long v = s_max[0];
        for (int q = 1; q < kWarps; ++q) v = v > s_max[q] ? v : s_max[q];
        atomicMax(&I.st->resp[0], v);
    }
    __syncthreads();
}

__global__ void __launch_bounds__(kThreads)
k_psi_loop_f64(const Inst* __restrict__ insts, int ninst, const Tile* __restrict__ tiles, int ntiles, LoopState* loop,
               int first) {
    using T = double;
    __shared__ int s_word, s_big;
    __shared__ unsigned long long s_max[kWarps];
    __shared__ Inst s_inst;  // a round's barrier empties L1: the descriptor stays here
    const Inst& I = s_inst;
    int cur_inst = -1, R = 0, done = 1;
    uint32_t rt = 0;
    for (int round = first;; ++round) {
        const C2<T>* cur = nullptr;
        const C2<T>* rhs = nullptr;
        C2<T>* nxt = nullptr;
        unsigned long long rmax = 0ull, thr = 0ull;
        bool rnan = false, fresh = true;
        for (int it = blockIdx.x; it < ntiles; it += gridDim.x) {
            const Tile t = ninst == 1 ? Tile{0, it * kThreads} : tiles[it];
            if (fresh || t.inst != cur_inst) {
                if (!fresh && !done) flush_f64(I, rmax, rnan, s_max);
                // an instance's `done` changes only at the end of a round
                if (t.inst != cur_inst || ninst > 1) {
                    const InstState* st = insts[t.inst].st;
                    for (int w = threadIdx.x; w < (int)(sizeof(Inst) / 8); w += kThreads)
                        ((unsigned long long*)&s_inst)[w] = ((const unsigned long long*)(insts + t.inst))[w];
                    done = *(volatile const int*)&st->done;
                    R = *(volatile const int*)&st->rhs;
                    rt = *(volatile const uint32_t*)&st->rand_t;
                }
                if (threadIdx.x == 0) s_big = 0;
                cur_inst = t.inst;
                fresh = false;
                __syncthreads();
                cur = (const C2<T>*)I.psi[ring_of(R, round)];
                rhs = (const C2<T>*)I.psi[R];
                nxt = (C2<T>*)I.psi[ring_of(R, round + 1)];
                thr = I.thr_psi;
                rmax = 0ull;
                rnan = false;
            }
            const int n = t.n0 + (int)threadIdx.x;
            const Geo& g = I.g;
            if (done || n >= g.N) continue;
            const int Nx = g.Nx, j = n / Nx, i = n - j * Nx;
            const C2<T>* __restrict__ U = (const C2<T>*)I.U;
            const C2<T> z = cmk<T>(T(0), T(0));
            const bool lt = i > 0, rg = i + 1 < Nx, dn = j > 0, up = j + 1 < g.Ny;
            // psi was written by other SMs in the round before: no read-only loads
            const C2<T> pc = cur[n];
            const C2<T> pl = lt ? cur[n - 1] : z, pr = rg ? cur[n + 1] : z;
            const C2<T> pd = dn ? cur[n - Nx] : z, pu = up ? cur[n + Nx] : z;
            const C2<T> ua = __ldg(&U[2 * n]), ub = __ldg(&U[2 * n + 1]);
            const C2<T> ual = lt ? __ldg(&U[2 * n - 2]) : z, ubd = dn ? __ldg(&U[2 * (n - Nx) + 1]) : z;
            const unsigned cd = (unsigned)__ldg(&I.code[n]);
            C2<T> rq = rhs[n];
            if (I.lang_psi_on) {
                const T lc = gsel<T>(I.lang_psi, I.flang_psi);
                rq.x = add_noise<T>(rq.x, lc, rand_1<T>((uint32_t)n, rt));
                rq.y = add_noise<T>(rq.y, lc, rand_2<T>((uint32_t)n, rt));
            }
            // the first sweep of a step stores the diagonal's reciprocal for the others
            T* dinv = (T*)I.dinv;
            T inv;
            if (round > 0) {
                inv = dinv[n];
            } else {
                const T* eps_sp = (const T*)I.eps_sp;
                const T eps = eps_sp ? __ldg(&eps_sp[n]) : gsel<T>(I.epsilon, I.fepsilon);
                inv = (cd & 3u) ? psi_diag_inv<T>(rq, eps, cd, gsel<T>(I.dt, I.fdt), GT(g, idx2), GT(g, idy2)) : T(0);
                dinv[n] = inv;
            }
            const C2<T> out = psi_node<T>(pl, pr, pd, pu, ual, ua, ubd, ub, rq, inv, cd);
            nxt[n] = out;
            // a NaN component counts as 0 (the reference's int conversion); magnitudes are
            // compared as integers, off the FP64 pipe.  A difference that overflows or is
            // NaN needs an operand beyond 2^1022.
            const unsigned big = max(max((unsigned)__double2hiint(out.x) & 0x7fffffffu, (unsigned)__double2hiint(out.y) & 0x7fffffffu),
                                     max((unsigned)__double2hiint(pc.x) & 0x7fffffffu, (unsigned)__double2hiint(pc.y) & 0x7fffffffu));
            if (__any_sync(__activemask(), *(volatile int*)&s_big == 0 || big >= 0x7fd00000u)) {
                const unsigned long long kAbs = 0x7fffffffffffffffull, kInf = 0x7ff0000000000000ull;
                unsigned long long bx = (unsigned long long)__double_as_longlong(out.x - pc.x) & kAbs;
                unsigned long long by = (unsigned long long)__double_as_longlong(out.y - pc.y) & kAbs;
                if ((bx > kInf) | (by > kInf)) rnan = true;
                bx = bx > kInf ? 0ull : bx;
                by = by > kInf ? 0ull : by;
                const unsigned long long m = bx > by ? bx : by;
                rmax = rmax > m ? rmax : m;
                if (rmax > thr) *(volatile int*)&s_big = 1;
            }
        }
        if (!fresh && !done) flush_f64(I, rmax, rnan, s_max);
        if (!end_round(insts, ninst, loop, round - first + 1, s_word, ClosePsi<1>{round, first, kFuse * min(loop->guard, kLoopGuard)}))
            break;
    }
}

// FP32: K = 3 sweeps per round.  A warp owns a strip of kWideCols = 56 output columns
// and the item's rows: each lane holds two adjacent columns, the 64 of them x0 - 4 .. x0 + 59,
// and sweep l (1..K) is valid l columns inside that, so the halo is recomputed in
// registers instead of being exchanged.  The warp walks down the rows: at step s it loads
// row j0-K+s of psi^(k) and the per-row inputs one row behind, and sweep l produces row
// j0-K+s-l from the three newest rows of sweep l-1 (each level lags the previous one by a
// row).  The x neighbours are the lane's other column and the adjacent lanes'.  The
// rows come through a ring of stages in shared memory that every lane fills for itself
// (asynchronous copies, three rows ahead, no barrier: a lane reads only what it copied).
// Of a round only the last sweep is stored, or all where the step before stopped inside
// the round; a stop elsewhere repeats the round up to there.
// What bounds it: latency, at 12 warps per SM (168 registers); 25 M warp instructions a
// round at 2049^2 where strips of 32 columns, one a lane, took 37 M.  A round at 2049^2:
// 54 us from a flushed L2 (60 as a timed launch), against 78 for a timed launch of those
// strips, which also held their rows in registers two ahead; 79 with two columns a lane
// and rows one ahead in registers.  Tiles of 64 x 32 nodes in shared memory, a column of
// 8 nodes a thread: 66 us with bulk copies for the next tile (the copy engine takes 60
// cycles for each of the short rows), 79 with plain loads, 90 with asynchronous copies.
constexpr int kPsiThreads = 64, kPsiWarps = kPsiThreads / 32;
constexpr int kWideMinB = 6;  // CTAs per SM that the registers must allow (7: spills)
// the reciprocal diagonal of a node without an x link (psi stays 0 there): a NaN that no
// arithmetic produces; the table holds the bits ^ kDead, so that 0 stands for it
constexpr unsigned kDead = 0xffffdeadu;

// A row's inputs of a lane's two nodes.
struct WideRow {
    float2 ua[2], ub[2], rq[2];
    float inv[2];
};

// A warp's residual maxima of a round into the instance's words.
template <int K = kFuse>
__device__ __forceinline__ void strip_flush(const Inst& I, const float (&wmax)[kFuse], const float (&wnan)[kFuse]) {
#pragma unroll
    for (int l = 0; l < K; ++l) {
        const unsigned m = __reduce_max_sync(0xffffffffu, __float_as_uint(wmax[l]));
        const bool nn = __any_sync(0xffffffffu, isnan(wnan[l]));
        if ((threadIdx.x & 31) == 0) {
            atomicMax(&I.st->resp[l], (unsigned long long)m);
            if (nn) atomicOr(&I.st->nanlv, 1 << l);
        }
    }
}

__device__ __forceinline__ float2 shfl_up2(float2 v) {
    return make_float2(__shfl_up_sync(0xffffffffu, v.x, 1), __shfl_up_sync(0xffffffffu, v.y, 1));
}
__device__ __forceinline__ float2 shfl_down2(float2 v) {
    return make_float2(__shfl_down_sync(0xffffffffu, v.x, 1), __shfl_down_sync(0xffffffffu, v.y, 1));
}

// Copy of B bytes into shared memory (zeros where take is false), in the thread's
// running group of copies; a group ends with copy_async_commit.
template <int B> __device__ __forceinline__ void copy_async(void* dst, const void* src, bool take) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], %2, %3;" ::"r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src), "n"(B),
                 "r"(take ? B : 0)
                 : "memory");
}
__device__ __forceinline__ void copy_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
// waits until at most N of the thread's groups are still on their way
template <int N> __device__ __forceinline__ void copy_async_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

// A row on its way: psi of a row and the other inputs of the row above it.  Every lane
// copies and reads its own two columns.
struct WideStage {
    float4 psi[32], rhs[32], U[2][32];
    uint2 inv[32];
};
constexpr int kWideStages = 4;

__global__ void __launch_bounds__(kPsiThreads, kWideMinB)
k_psi_loop_f32(const Inst* __restrict__ insts, int ninst, const Item* __restrict__ items, int nitems, LoopState* loop,
               int first) {
    constexpr int K = kFuse, NS = kWideStages;
    static_assert(K + 1 == NS, "the walk's windows turn with the stages");
    __shared__ WideStage s_st[kPsiWarps][NS];
    __shared__ int s_word;
    const int lane = threadIdx.x & 31;
    WideStage* const st4 = s_st[threadIdx.x >> 5];
    const int gw = blockIdx.x * kPsiWarps + (threadIdx.x >> 5), nw = gridDim.x * kPsiWarps;
    const float2 z = make_float2(0.f, 0.f);
    for (int round = first;; ++round) {
        int cur_inst = -1, done = 1;
        float wmax[K], wnan[K];  // running maxima of the differences: one drops NaN, one keeps it
        const float2* cur = nullptr;
        const float2* rhs = nullptr;
        float2* outb[K];
        uint32_t rt = 0;
        for (int it = gw; it < nitems; it += nw) {
            // odd rounds walk backwards: what a round used last is still in L2
            const Item w = items[(round & 1) ? nitems - 1 - it : it];
            if (w.inst != cur_inst) {
                if (cur_inst >= 0 && !done) strip_flush(insts[cur_inst], wmax, wnan);
                cur_inst = w.inst;
                // an instance's loop state changes only at the end of a round
                const Inst& I = insts[cur_inst];
                const InstState* st = I.st;
                done = *(volatile const int*)&st->done;
                const int R = *(volatile const int*)&st->rhs;
                const int redo = *(volatile const int*)&st->redo, keep = *(volatile const int*)&st->keep;
                const int r0 = redo ? round - 1 : round;  // finished rounds that this one starts from
                rt = *(volatile const uint32_t*)&st->rand_t;
                cur = (const float2*)I.psi[ring_of(R, r0)];
                rhs = (const float2*)I.psi[R];
#pragma unroll
                for (int l = 0; l < K; ++l) {
                    const bool kept = redo ? l + 1 == redo : (l + 1 == K || keep);
                    outb[l] = kept ? (float2*)I.psi[l + 1 == K ? ring_of(R, r0 + 1) : mid_of(R, l + 1)] : nullptr;
                    wmax[l] = wnan[l] = 0.f;
                }
            }
            if (done) continue;
            const Inst& I = insts[cur_inst];
            const int Nx = I.g.Nx, Ny = I.g.Ny;
            const float4* __restrict__ U = (const float4*)I.U;
            float* dinv = (float*)I.dinv;
            const bool lang = I.lang_psi_on != 0;
            const int i0 = w.x0 - 4 + 2 * lane, j0 = w.j0, rows = w.pad, S = rows + 2 * K;
            const bool in0 = i0 >= 0 && i0 < Nx, in1 = i0 + 1 >= 0 && i0 + 1 < Nx;
            const bool own0 = in0 && lane >= 2 && lane <= 29, own1 = in1 && lane >= 2 && lane <= 29;
            // step s uses psi of row j0 - K + s and the other inputs of the row above
            auto issue = [&](int s, WideStage& t) {
                const int y = j0 - K + s, n = i0 + Nx * y;
                const bool row = y >= 0 && y < Ny && s < S, up = y >= 1 && y <= Ny && s < S;
                copy_async<8>(&t.psi[lane].x, cur + (row && in0 ? n : 0), row && in0);
                copy_async<8>(&t.psi[lane].z, cur + (row && in1 ? n + 1 : 0), row && in1);
                const int m0 = up && in0 ? n - Nx : 0, m1 = up && in1 ? n - Nx + 1 : 0;
                copy_async<8>(&t.rhs[lane].x, rhs + m0, up && in0);
                copy_async<8>(&t.rhs[lane].z, rhs + m1, up && in1);
                copy_async<16>(&t.U[0][lane], U + m0, up && in0);
                copy_async<16>(&t.U[1][lane], U + m1, up && in1);
                if (round > 0) {
                    copy_async<4>(&t.inv[lane].x, dinv + m0, up && in0);
                    copy_async<4>(&t.inv[lane].y, dinv + m1, up && in1);
                }
                copy_async_commit();
            };
            // window of sweep l-1 (l = 1..K) as seen by sweep l: rows y-1 and y
            float2 wp[K][2], wc[K][2];
            WideRow D[K + 1];  // D[m]: inputs of row (j0 - K + s - 1) - m
#pragma unroll
            for (int l = 0; l < K; ++l) wp[l][0] = wp[l][1] = wc[l][0] = wc[l][1] = z;
#pragma unroll
            for (int m = 0; m <= K; ++m)
#pragma unroll
                for (int c = 0; c < 2; ++c) {
                    D[m].ua[c] = D[m].ub[c] = D[m].rq[c] = z;
                    D[m].inv[c] = __uint_as_float(kDead);
                }
#pragma unroll
            for (int a = 0; a < NS - 1; ++a) issue(a, st4[a]);
            // one step of the walk; head: sweep l starts at step 2l (earlier rows are above
            // its halo), later steps do all sweeps
            auto step = [&](int s, WideStage& t, WideStage& tn, auto head) {
                constexpr bool kHead = decltype(head)::value;
                copy_async_wait<NS - 2>();
                const float4 pv = t.psi[lane], rv = t.rhs[lane], u0 = t.U[0][lane], u1 = t.U[1][lane];
                float2 newrow[2] = {make_float2(pv.x, pv.y), make_float2(pv.z, pv.w)};
#pragma unroll
                for (int m = K; m >= 1; --m) D[m] = D[m - 1];
                WideRow& q = D[0];
                q.ua[0] = make_float2(u0.x, u0.y);
                q.ub[0] = make_float2(u0.z, u0.w);
                q.ua[1] = make_float2(u1.x, u1.y);
                q.ub[1] = make_float2(u1.z, u1.w);
                q.rq[0] = make_float2(rv.x, rv.y);
                q.rq[1] = make_float2(rv.z, rv.w);
                const int yd = j0 - K + s - 1;
                if (lang || round == 0) {  // (uniform)
                    const bool row = yd >= 0 && yd < Ny;
                    const int n = i0 + Nx * yd;
                    const float* eps_sp = (const float*)I.eps_sp;
#pragma unroll
                    for (int c = 0; c < 2; ++c) {
                        const bool ld = row && (c ? in1 : in0);
                        if (lang && ld) {
                            q.rq[c].x = add_noise<float>(q.rq[c].x, I.flang_psi, rand_1<float>((uint32_t)(n + c), rt));
                            q.rq[c].y = add_noise<float>(q.rq[c].y, I.flang_psi, rand_2<float>((uint32_t)(n + c), rt));
                        }
                        if (round == 0) {  // the diagonal's reciprocals, stored for the step's later rounds
                            const unsigned cd = ld ? (unsigned)__ldg(&I.code[n + c]) : 0u;
                            float v = __uint_as_float(kDead);
                            if (cd & 3u)
                                v = psi_diag_inv<float>(q.rq[c], eps_sp ? __ldg(&eps_sp[n + c]) : I.fepsilon, cd, I.fdt, I.g.fidx2,
                                                        I.g.fidy2);
                            if ((c ? own1 : own0) && yd >= j0 && yd < j0 + rows) dinv[n + c] = __uint_as_float(__float_as_uint(v) ^ kDead);
                            q.inv[c] = v;
                        }
                    }
                }
                if (round > 0) {
                    const uint2 iv = t.inv[lane];
                    q.inv[0] = __uint_as_float(iv.x ^ kDead);
                    q.inv[1] = __uint_as_float(iv.y ^ kDead);
                }
                issue(s + NS - 1, tn);  // into the stage that the step before has read
#pragma unroll
                for (int l = 1; l <= K; ++l) {
                    float2 out[2] = {z, z};
                    if (!kHead || s >= 2 * l) {
                        const float2 p0 = wc[l - 1][0], p1 = wc[l - 1][1];
                        const WideRow& d = D[l - 1];
                        const float2 pl = shfl_up2(p1), pr = shfl_down2(p0), ual = shfl_up2(d.ua[1]);
                        // every lane computes: outside the domain the inputs are zero and dead,
                        // and psi_node returns 0 there
                        out[0] = psi_node<float>(pl, p1, wp[l - 1][0], newrow[0], ual, d.ua[0], D[l].ub[0], d.ub[0], d.rq[0],
                                                 d.inv[0], __float_as_uint(d.inv[0]) != kDead ? 1u : 0u);
                        out[1] = psi_node<float>(p0, pr, wp[l - 1][1], newrow[1], d.ua[0], d.ua[1], D[l].ub[1], d.ub[1], d.rq[1],
                                                 d.inv[1], __float_as_uint(d.inv[1]) != kDead ? 1u : 0u);
                        // rows K .. K + rows - 1 of the walk are the strip's own
                        if (s - l >= K && s - l < K + rows) {
                            const float dx0 = out[0].x - p0.x, dy0 = out[0].y - p0.y, dx1 = out[1].x - p1.x, dy1 = out[1].y - p1.y;
                            // a NaN component counts as 0 (the reference's int conversion); nodes
                            // outside the domain stay 0
                            asm("max.abs.f32 %0, %0, %1, %2;" : "+f"(wmax[l - 1]) : "f"(dx0), "f"(dy0));
                            asm("max.NaN.abs.f32 %0, %0, %1, %2;" : "+f"(wnan[l - 1]) : "f"(dx0), "f"(dy0));
                            asm("max.abs.f32 %0, %0, %1, %2;" : "+f"(wmax[l - 1]) : "f"(dx1), "f"(dy1));
                            asm("max.NaN.abs.f32 %0, %0, %1, %2;" : "+f"(wnan[l - 1]) : "f"(dx1), "f"(dy1));
                            if (outb[l - 1]) {
                                float2* o = outb[l - 1] + (i0 + Nx * (j0 - K + s - l));
                                if (own0) o[0] = out[0];
                                if (own1) o[1] = out[1];
                            }
                        }
                    }
                    // sweep l has used the window of sweep l-1: advance it by one row
#pragma unroll
                    for (int c = 0; c < 2; ++c) {
                        wp[l - 1][c] = wc[l - 1][c];
                        wc[l - 1][c] = newrow[c];
                        newrow[c] = out[c];
                    }
                }
            };
            int s = 0;
            for (; s < 2 * NS; s += NS) {
#pragma unroll
                for (int a = 0; a < NS; ++a) step(s + a, st4[a], st4[(a + NS - 1) % NS], std::true_type{});
            }
            for (; s < S; s += NS) {
#pragma unroll
                for (int a = 0; a < NS; ++a) step(s + a, st4[a], st4[(a + NS - 1) % NS], std::false_type{});
            }
            copy_async_wait<0>();
            // the halo lanes' columns are other strips'
            if (lane < 2 || lane > 29)
#pragma unroll
                for (int l = 0; l < K; ++l) wmax[l] = wnan[l] = 0.f;
        }
        if (cur_inst >= 0 && !done) strip_flush(insts[cur_inst], wmax, wnan);
        if (!end_round(insts, ninst, loop, round - first + 1, s_word, ClosePsi<K>{round, first, kFuse * min(loop->guard, kLoopGuard)}))
            break;
    }
}

// The Jacobi loop of the A step (svirl/cuda/td.h:310-463) in one cooperative launch, FP32,
// two sweeps per round.  It iterates the offset delta = A - A^(0) from the loop's
// right-hand side: with A^(k) = A^(0) + delta^(k) the update of a link is
//   delta' = (noise + dt rho (js + rh) + dt rho k2 (dd nbs(A^(0)) - 2 d^-2 A^(0))
//            + dt rho k2 dd nbs(delta^(k))) / D,
// and the stop rule's |A^(k+1) - A^(k)| = |delta^(k+1) - delta^(k)|.  In FP32 the iterates of
// A itself differ by whole units in the last place once |A| > 8 (the Landau gauge reaches
// H L), which the absolute stop rule of 1e-6 (svirl/solvers/td.py:53-57) never accepts;
// delta is small, so the loop converges.  The division by a link's constant diagonal is a
// multiplication by its reciprocal.
// The fixed part X of an update takes the supercurrent phase from delta^(2 floor(k/2)) (the
// reference's aliasing, td.cu), so a round's two sweeps share it and it stays in
// registers: one pass over A^(0), delta and psi.
// Strips as in k_psi_loop_f32: two columns a lane, 64 columns x0 - 2 .. x0 + 61 of which 60
// are the strip's own, rows through a ring of asynchronous copies.  At a step the row y is
// new: X and the first sweep of row y - 1, the second sweep of row y - 2.
// A round stores the sweep after which the loop stopped a step ago, if that is its first,
// else its second; a loop that stops or goes on elsewhere repeats the round (redo: 1 or 2
// to stop after that sweep, 3 to go on).
// Two sweeps at 2049^2, kappa 4, from a flushed L2: 87 us; as a launch per sweep, with X
// stored and read back and a thread per node that loads its twelve neighbours (531
// instructions a node in the first of a pair), 158.
struct AStage {
    float2 a0[32], b0[32], da[32], db[32];
    float4 psi[32];
};
// A row of link values of a lane's two columns, with the neighbours' left and right of them.
struct ARow {
    float a[2], b[2], aL, bL, bR;
};
__device__ __forceinline__ void row_sides(ARow& r) {
    r.aL = __shfl_up_sync(0xffffffffu, r.a[1], 1);
    r.bL = __shfl_up_sync(0xffffffffu, r.b[1], 1);
    r.bR = __shfl_down_sync(0xffffffffu, r.b[0], 1);
}
__device__ __forceinline__ float row_nbs_x(float idy2, float idxy, const ARow& dn, const ARow& cu, const ARow& up, int c) {
    return A_nbs_x<float>(idy2, idxy, dn.a[c], up.a[c], dn.b[c], c == 0 ? dn.b[1] : dn.bR, cu.b[c], c == 0 ? cu.b[1] : cu.bR);
}
__device__ __forceinline__ float row_nbs_y(float idx2, float idxy, const ARow& cu, const ARow& up, int c) {
    return A_nbs_y<float>(idx2, idxy, c == 0 ? cu.bL : cu.b[0], c == 0 ? cu.b[1] : cu.bR, c == 0 ? cu.aL : cu.a[0],
                          c == 0 ? up.aL : up.a[0], cu.a[c], up.a[c]);
}

// Buffer of delta^(k), k even and positive, of a loop with A^(0) in buffer R.
__device__ __forceinline__ int delta_of(int R, int k) { return (R + 1 + ((k / 2 - 1) & 1)) % 3; }

struct CloseA {
    int guard;  // in sweeps
    int once;   // a timed loop: one round
    __device__ __forceinline__ int operator()(const Inst& I, InstState* st) const {
        const int R = *(volatile const int*)&st->rhsA, redo = *(volatile const int*)&st->redo, k = *(volatile const int*)&st->sweep;
        const int stored = *(volatile const int*)&st->keep;  // the sweep that the round stored
        int stop = redo == 3 ? 0 : redo, go = redo == 3;
        if (!redo) {
            stop = stop_level<2>(st, k, I.thr_A, guard);
            if (once || (!stop && k + 2 >= guard)) return 3;
            if (stop != stored && (stop || stored != 2)) {
                st->redo = stop ? stop : 3;
                return 1;
            }
            go = !stop;
        }
        st->redo = 0;
        if (go) {
            st->sweep = k + 2;
            st->keep = *(volatile const int*)&st->last_sweeps_A == k + 3 ? 1 : 2;
            return 1;
        }
        const int s = k + stop;
        st->sweep = s;
        st->done = 1;
        st->commitA = 1 + R;  // the buffers hold offsets from A^(0); k_A_commit adds it
        st->rhsA = delta_of(R, k + 2);
        st->last_sweeps_A = s;
        st->total_sweeps_A += s;
        if (s > st->max_sweeps_A) st->max_sweeps_A = s;
        return 0;
    }
};

constexpr int kAMinB = 6;  // CTAs per SM that the registers must allow (7: spills, 56 us a sweep against 43)
__global__ void __launch_bounds__(kPsiThreads, kAMinB)
k_A_loop_f32(const Inst* __restrict__ insts, int ninst, const Item* __restrict__ items, int nitems, LoopState* loop, int once) {
    constexpr int NS = kWideStages;
    __shared__ AStage s_st[kPsiWarps][NS];
    __shared__ int s_word;
    const int lane = threadIdx.x & 31;
    AStage* const st4 = s_st[threadIdx.x >> 5];
    const int gw = blockIdx.x * kPsiWarps + (threadIdx.x >> 5), nw = gridDim.x * kPsiWarps;
    for (int seq = 1;; ++seq) {
        int cur_inst = -1, done = 1, k = 0, R = 0, keep_at = 2;
        bool quiet = false;  // a repeated round: its residuals are known
        uint32_t rt = 0;
        float wmax[kFuse], wnan[kFuse];
        for (int it = gw; it < nitems; it += nw) {
            const Item w = items[(seq & 1) ? it : nitems - 1 - it];
            if (w.inst != cur_inst) {
                if (cur_inst >= 0 && !done && !quiet) strip_flush<2>(insts[cur_inst], wmax, wnan);
                cur_inst = w.inst;
                // an instance's loop state changes only at the end of a round
                const InstState* st = insts[cur_inst].st;
                done = *(volatile const int*)&st->done;
                k = *(volatile const int*)&st->sweep;
                R = *(volatile const int*)&st->rhsA;
                const int redo = *(volatile const int*)&st->redo;
                quiet = redo != 0;
                keep_at = redo ? (redo == 1 ? 1 : 2) : *(volatile const int*)&st->keep;
                rt = *(volatile const uint32_t*)&st->rand_t;
                wmax[0] = wmax[1] = wnan[0] = wnan[1] = 0.f;
            }
            if (done) continue;
            const Inst& I = insts[cur_inst];
            const int Nx = I.g.Nx, Ny = I.g.Ny, Nxa = Nx - 1, Na = I.g.Na;
            const float* __restrict__ base = (const float*)I.ab[R];
            const float* cur = (const float*)I.ab[k == 0 ? R : delta_of(R, k)];  // k = 0: not read
            const float* vpi = (const float*)I.vpi;
            float* out = (float*)I.ab[delta_of(R, k + 2)];
            const float2* __restrict__ psi = (const float2*)I.psi[*(volatile const int*)&I.st->rhs];
            const float k2 = I.fkappa2, dt_rho = I.fdt * I.frho, dt_rho_k2 = dt_rho * k2, H = I.fH;
            const float idx = I.g.fidx, idy = I.g.fidy, idx2 = I.g.fidx2, idy2 = I.g.fidy2, idxy = I.g.fidxy, dx = I.g.fdx, dy = I.g.fdy;
            const float c2 = I.fdt * I.frho * I.fkappa2;
            const float rden_a = 1.f / (1.f + 2.f * c2 * idy2), rden_b = 1.f / (1.f + 2.f * c2 * idx2);
            const bool lang = I.lang_A_on != 0;
            const float lc = I.flang_A;
            const int i0 = w.x0 - 2 + 2 * lane, j0 = w.j0, rows = w.pad, S = rows + 4;
            const bool in[2] = {i0 >= 0 && i0 < Nx, i0 + 1 >= 0 && i0 + 1 < Nx};    // node, and its y link's column
            const bool ina[2] = {i0 >= 0 && i0 < Nxa, i0 + 1 >= 0 && i0 + 1 < Nxa};  // x link's column
            const bool own = lane >= 1 && lane <= 30;
            auto issue = [&](int s, AStage& t) {
                const int y = j0 - 2 + s;
                const bool row = y >= 0 && y < Ny && s < S, rowb = y >= 0 && y < Ny - 1 && s < S;
#pragma unroll
                for (int c = 0; c < 2; ++c) {
                    const bool ta = row && ina[c], tb = rowb && in[c], tp = row && in[c];
                    const int la = ta ? i0 + c + Nxa * y : 0, lb = tb ? Na + i0 + c + Nx * y : 0;
                    copy_async<4>(c ? &t.a0[lane].y : &t.a0[lane].x, base + la, ta);
                    copy_async<4>(c ? &t.b0[lane].y : &t.b0[lane].x, base + lb, tb);
                    copy_async<4>(c ? &t.da[lane].y : &t.da[lane].x, cur + la, ta && k > 0);
                    copy_async<4>(c ? &t.db[lane].y : &t.db[lane].x, cur + lb, tb && k > 0);
                    copy_async<8>(c ? &t.psi[lane].z : &t.psi[lane].x, psi + (tp ? i0 + c + Nx * y : 0), tp);
                }
                copy_async_commit();
            };
            // link-weight bits of the row above the new one, fetched with it
            auto codes = [&](int s) -> unsigned {
                const int y = j0 - 3 + s;
                unsigned cd = 0u;
                if (y >= 0 && y < Ny && s < S) {
                    if (in[0]) cd = __ldg(&I.code[i0 + Nx * y]);
                    if (in[1]) cd |= (unsigned)__ldg(&I.code[i0 + 1 + Nx * y]) << 8;
                }
                return cd;
            };
            const ARow zr = {{0.f, 0.f}, {0.f, 0.f}, 0.f, 0.f, 0.f};
            // rows y - 1 and y - 2 of A^(0) and delta^(k); y - 2 and y - 3 of the first sweep
            ARow A1 = zr, A2 = zr, D1 = zr, D2 = zr, F1 = zr, F2 = zr;
            float2 P1[2] = {make_float2(0.f, 0.f), make_float2(0.f, 0.f)};
            float xa2[2] = {0.f, 0.f}, xb2[2] = {0.f, 0.f};  // X of row y - 2
            unsigned cdr[NS];
#pragma unroll
            for (int a = 0; a < NS - 1; ++a) {
                issue(a, st4[a]);
                cdr[a] = codes(a);
            }
            auto step = [&](int s, AStage& t, AStage& tn, unsigned cd) {
                copy_async_wait<NS - 2>();
                const int y = j0 - 2 + s;
                ARow A0, D0;
                const float2 va = t.a0[lane], vb = t.b0[lane], wa = t.da[lane], wb = t.db[lane];
                A0.a[0] = va.x; A0.a[1] = va.y; A0.b[0] = vb.x; A0.b[1] = vb.y;
                D0.a[0] = wa.x; D0.a[1] = wa.y; D0.b[0] = wb.x; D0.b[1] = wb.y;
                const float4 pv = t.psi[lane];
                const float2 P0[2] = {make_float2(pv.x, pv.y), make_float2(pv.z, pv.w)};
                issue(s + NS - 1, tn);  // into the stage that the step before has read
                row_sides(A0);
                row_sides(D0);
                const float2 pr = make_float2(__shfl_down_sync(0xffffffffu, P1[0].x, 1), __shfl_down_sync(0xffffffffu, P1[0].y, 1));
                // X and the first sweep of row j
                const int j = y - 1;
                float xa[2] = {0.f, 0.f}, xb[2] = {0.f, 0.f};
                ARow F0 = zr;
                if (j >= 0 && j < Ny) {
                    const bool edge = j == 0 || j == Ny - 1;
                    const float dda = edge ? 2.f : 1.f;
                    const float rha = j == 0 ? 2.f * k2 * H * idy : (j == Ny - 1 ? -2.f * k2 * H * idy : 0.f);
#pragma unroll
                    for (int c = 0; c < 2; ++c) {
                        const int i = i0 + c;
                        const float ddb = i == 0 || i == Nx - 1 ? 2.f : 1.f;
                        const float rhb = i == 0 ? -2.f * k2 * H * idx : (i == Nx - 1 ? 2.f * k2 * H * idx : 0.f);
                        float pa = A1.a[c] + D1.a[c], pb = A1.b[c] + D1.b[c], fa = 0.f, fb = 0.f;
                        const bool ha = ina[c], hb = in[c] && j < Ny - 1;
                        if (vpi) {
                            pa = ha ? vpi[i + Nxa * j] : 0.f;
                            pb = hb ? vpi[Na + i + Nx * j] : 0.f;
                        }
                        if (lang) {
                            fa = add_noise<float>(0.f, lc, rand_1<float>((uint32_t)(i + Nxa * j), rt));
                            fb = add_noise<float>(0.f, lc, rand_2<float>((uint32_t)(Na + i + Nx * j), rt));
                        }
                        const float ja = mul_rn<float>(idx, js_of<float>(P1[c], dx * pa, c == 0 ? P1[1] : pr));
                        const float jb = mul_rn<float>(idy, js_of<float>(P1[c], dy * pb, P0[c]));
                        xa[c] = A_fixed<float>(fa, dt_rho, (cd >> (8 * c)) & 2u ? ja : 0.f, rha) +
                                A_base<float>(dt_rho_k2, dda, row_nbs_x(idy2, idxy, A2, A1, A0, c), idy2, A1.a[c]);
                        xb[c] = A_fixed<float>(fb, dt_rho, (cd >> (8 * c)) & 8u ? jb : 0.f, rhb) +
                                A_base<float>(dt_rho_k2, ddb, row_nbs_y(idx2, idxy, A1, A0, c), idx2, A1.b[c]);
                        const float na = fma(dt_rho_k2 * dda, row_nbs_x(idy2, idxy, D2, D1, D0, c), xa[c]) * rden_a;
                        const float nb = fma(dt_rho_k2 * ddb, row_nbs_y(idx2, idxy, D1, D0, c), xb[c]) * rden_b;
                        F0.a[c] = ha ? na : 0.f;
                        F0.b[c] = hb ? nb : 0.f;
                    }
                }
                row_sides(F0);
                // the second sweep of row j - 1
                float ga[2] = {0.f, 0.f}, gb[2] = {0.f, 0.f};
                if (j >= 1 && j - 1 < Ny) {
                    const float dda = j == 1 || j == Ny ? 2.f : 1.f;
#pragma unroll
                    for (int c = 0; c < 2; ++c) {
                        const int i = i0 + c;
                        const float ddb = i == 0 || i == Nx - 1 ? 2.f : 1.f;
                        const float na = fma(dt_rho_k2 * dda, row_nbs_x(idy2, idxy, F2, F1, F0, c), xa2[c]) * rden_a;
                        const float nb = fma(dt_rho_k2 * ddb, row_nbs_y(idx2, idxy, F1, F0, c), xb2[c]) * rden_b;
                        ga[c] = ina[c] ? na : 0.f;
                        gb[c] = in[c] && j < Ny ? nb : 0.f;
                    }
                }
                // rows 2 .. rows + 1 of the walk are the strip's own
                auto tell = [&](int l, float d0, float d1) {
                    asm("max.abs.f32 %0, %0, %1, %2;" : "+f"(wmax[l]) : "f"(d0), "f"(d1));
                    asm("max.NaN.abs.f32 %0, %0, %1, %2;" : "+f"(wnan[l]) : "f"(d0), "f"(d1));
                };
                auto store = [&](int yy, const float (&va2)[2], const float (&vb2)[2]) {
#pragma unroll
                    for (int c = 0; c < 2; ++c) {
                        if (own && ina[c]) out[i0 + c + Nxa * yy] = va2[c];
                        if (own && in[c] && yy < Ny - 1) out[Na + i0 + c + Nx * yy] = vb2[c];
                    }
                };
                if (s >= 3 && s < rows + 3) {
                    tell(0, F0.a[0] - D1.a[0], F0.a[1] - D1.a[1]);
                    tell(0, F0.b[0] - D1.b[0], F0.b[1] - D1.b[1]);
                    if (keep_at == 1) store(j, F0.a, F0.b);
                }
                if (s >= 4 && s < rows + 4) {
                    tell(1, ga[0] - F1.a[0], ga[1] - F1.a[1]);
                    tell(1, gb[0] - F1.b[0], gb[1] - F1.b[1]);
                    if (keep_at == 2) store(j - 1, ga, gb);
                }
                A2 = A1;
                A1 = A0;
                D2 = D1;
                D1 = D0;
                F2 = F1;
                F1 = F0;
#pragma unroll
                for (int c = 0; c < 2; ++c) {
                    P1[c] = P0[c];
                    xa2[c] = xa[c];
                    xb2[c] = xb[c];
                }
            };
            for (int s = 0; s < S; s += NS) {
#pragma unroll
                for (int a = 0; a < NS; ++a) {
                    cdr[(a + NS - 1) % NS] = codes(s + a + NS - 1);
                    step(s + a, st4[a], st4[(a + NS - 1) % NS], cdr[a]);
                }
            }
            copy_async_wait<0>();
            if (!own) wmax[0] = wmax[1] = wnan[0] = wnan[1] = 0.f;  // the halo lanes' columns are other strips'
        }
        if (cur_inst >= 0 && !done && !quiet) strip_flush<2>(insts[cur_inst], wmax, wnan);
        if (!end_round(insts, ninst, loop, seq, s_word, CloseA{min(loop->guard, kLoopGuard), once})) break;
    }
}

// The loop's kernel: FP64 over tiles (Tile), FP32 over the items of strips.
const void* psi_loop_fn(int dtype) { return dtype == 8 ? (const void*)k_psi_loop_f64 : (const void*)k_psi_loop_f32; }
int psi_loop_threads(int dtype) { return dtype == 8 ? kThreads : kPsiThreads; }

const void* A_loop_fn() { return (const void*)k_A_loop_f32; }

// CTAs of a loop kernel that are resident at once.
static int loop_cap(const void* fn, int threads) {
    int dev = 0, sms = 1, per_sm = 1;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, fn, threads, 0) != cudaSuccess || per_sm < 1) per_sm = 1;
    return sms * per_sm;
}

// CTAs of the loop over n tiles or items.
int psi_loop_grid(int dtype, int n) {
    const int need = dtype == 8 ? n : (n + kPsiWarps - 1) / kPsiWarps, cap = loop_cap(psi_loop_fn(dtype), psi_loop_threads(dtype));
    return need < cap ? need : cap;
}
int A_loop_grid(int n) {
    const int need = (n + kPsiWarps - 1) / kPsiWarps, cap = loop_cap(A_loop_fn(), kPsiThreads);
    return need < cap ? need : cap;
}

// Strip height of an FP32 loop for a set of instances: a round lasts as long as the warp
// with the most items, ceil(items / warps), and an item of R rows costs about R + halo
// steps.  R + 2 K steps are walked in fours.
// *cost: of the choice, in row steps.
static int choose_rows(const Geo* const* geos, int n, const void* fn, int cols, int K, long long* cost_out = nullptr) {
    int best = 0;
    long long best_cost = -1;
    const long long warps = (long long)loop_cap(fn, kPsiThreads) * kPsiWarps;
    for (int S = 12; S <= 68; S += kWideStages) {
        const int R = S - 2 * K;
        long long items = 0;
        for (int q = 0; q < n; ++q) items += (long long)((geos[q]->Nx + cols - 1) / cols) * ((geos[q]->Ny + R - 1) / R);
        const long long cost = (items + warps - 1) / warps * (long long)(R + K);
        if (best_cost < 0 || cost < best_cost) {
            best_cost = cost;
            best = R;
        }
    }
    if (cost_out) *cost_out = best_cost;
    return best;
}
int choose_loop_rows(const Geo* const* geos, int n) { return choose_rows(geos, n, psi_loop_fn(4), kWideCols, kFuse); }
int choose_A_rows(const Geo* const* geos, int n) { return choose_rows(geos, n, A_loop_fn(), kACols, 2); }

// A usual time step (22 psi sweeps, 3 to 4 A sweeps) of a batch of FP32 films by the loops
// here, us: launches, the rounds' row steps, the closing of every film's loop.  Fitted to 76
// batches of 2 to 600 films of 64^2 .. 760^2, measured 166 to 1370 us, within 12 %.
double loops_step_us(const Geo* const* geos, int n, bool any_A) {
    long long psi = 0, A = 0;
    choose_rows(geos, n, psi_loop_fn(4), kWideCols, kFuse, &psi);
    if (any_A) choose_rows(geos, n, A_loop_fn(), kACols, 2, &A);
    return 75.0 + 8.4 * (double)psi + 0.55 * n + (any_A ? 22.0 + 5.1 * (double)A : 0.0);
}

// Items of an instance for the FP32 loops, band by band (warps that run at the same time
// share halo rows in L2).
void add_loop_items(std::vector<Item>& items, const Geo& g, int inst, int rows, int cols) {
    for (int j0 = 0; j0 < g.Ny; j0 += rows)
        for (int x0 = 0; x0 < g.Nx; x0 += cols) items.push_back(Item{inst, x0, j0, std::min(rows, g.Ny - j0)});
}

}  // namespace glgpu
