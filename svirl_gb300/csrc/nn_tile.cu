// 3x3 convolutions for the shapes that the whole-row TMA kernels of nn_tc.cu do not
// take: channel counts that are not multiples of 64 (the network's full-resolution
// level has 8, 32 and 64 + 32) and images of any width.  tcgen05.mma with operands
// loaded by TMA, as there.
//
// Output tiles are 8 x 16 pixels (M = 128, TMEM lane = 8 ty + tx).  A stage holds one
// input-channel chunk of a tile with its halo: one TMA box of 16 x 18 pixels x 64
// channels (36 KB; ten of the sixteen columns are read, the rest make the rows a
// multiple of the eight-row swizzle group).  All nine taps are views of that box: the A
// descriptor of tap (ky, kx) starts ky rows of 2 KB and kx pixels of 128 bytes into it,
// and its eight-pixel groups (the tile's rows) are 2 KB apart.  So the activations cross
// from L2 2.25 times (1.4 times in columns that count) instead of nine times.  What the
// box holds outside the image or beyond the chunk's channels the copy engine fills with
// zeros, which is the "same" padding, and the channels in use take c / 16 K steps a tap.
// The weights of the CTA's output channels stay in shared memory.  The K steps run tap by
// tap and through all chunks of a tap, the order of the other kernels, so the sums are the
// same bitwise (a backward pass masks by the sign of what a forward pass stored).
//
// Eight input channels (the network's first layer): a pixel is one 16-byte row, a core
// matrix of the unswizzled layout is eight of a box's pixels, and a K step of 16 takes two
// taps, the second at the descriptor's leading offset (tap 9 is a block of zeros).
//
// What bounds it: the copy engine takes about five cycles per 128-byte row of a box,
// filled or not, 1440 cycles a box (MMAs alone: about 50 cycles each).  64 images of
// 128^2, us, thread-gather kernel / this one (copies of the input and output alone at the
// measured HBM rate): 8 -> 32 channels 201 / 31 (13), 32 -> 32 390 / 41 (20), 64 + 32 -> 32
// 966 / 90 (40), 32 -> 8 358 / 37 (13) (back to back; 10 us more each as single calls from a
// flushed L2); the 64 + 32 -> 32 layer forward and backward, 32 images: 1555 / 320.
#include <type_traits>

#include "nn_tc.cuh"

#include "../../include/glgpu.h"

namespace glnn_tc {

constexpr int TW = 8, TH = 16;                       // output pixels of a tile
constexpr int BOXW = 16, BOXH = TH + 2;              // pixels of an input box
constexpr int BOX_BYTES = BOXW * BOXH * 128;         // 36,864: a multiple of the swizzle atom's 1 KB
constexpr int ROW_BYTES = BOXW * 128;                // a box row
constexpr int TILE_THREADS = 192;                    // TMA warp, MMA warp, four epilogue warps
constexpr int ACC = 2;                               // accumulators in tensor memory
constexpr int SMEM_MAX = 227 * 1024;
constexpr int kTileStagesMax = 4;

struct TileShape {
    int nck1, nck, stages, smem;  // chunks of the first input, of both; operand stages
};
// eight channels: bytes of a box, of the zeros after the stages (as far as a view of tap 9
// reaches), and of a stage
constexpr int BOX8_BYTES = BOXW * BOXH * 16, ZERO8_BYTES = (TH - 1) * BOXW * 16 + TW * 16;

// A views of a box: the tile's rows, eight pixels each, are ROW_BYTES apart
constexpr uint32_t kBoxHi = desc_hi(ROW_BYTES), kWeightHi = desc_hi(1024);

template <int MODE> __device__ __forceinline__ constexpr uint32_t tap_off(int tap) {
    return (uint32_t)(((MODE == 0 ? tap / 3 : 2 - tap / 3) * ROW_BYTES + (MODE == 0 ? tap % 3 : 2 - tap % 3) * 128) >> 4);
}

// The MMAs of a tile, tap by tap and through the chunks of a tap: chunk c takes KS[c] K steps
// (ks[c] where that is 0) from the box at a[c]; w: the weights (low descriptor halves).  The
// operands are constants away from the bases, which a loop over chunks with a branch on
// their steps moved for every MMA.  64 images of 128^2 to 32 channels, us, by that loop /
// this: 32 + 32 189 / 81, 64 + 32 154 / 91, 64 + 48 181 / 101, 64 + 64 150 / 109, 96 183 / 91.
// One chunk unrolled over all taps, more over a row of taps (one chunk by rows: 48 against
// 46 us at 32 channels, 68 against 64 at 64; two unrolled over all taps: 97).
template <int MODE, int WB, int... KS>
__device__ __forceinline__ void tile_mmas(uint32_t d, const uint32_t (&a)[sizeof...(KS)], const int (&ks)[sizeof...(KS)],
                                          uint32_t w, uint32_t idesc) {
    constexpr int kSteps[] = {KS...}, NCK = sizeof...(KS);
    if constexpr (NCK == 1) {
#pragma unroll
        for (int tap = 0; tap < 9; ++tap)
#pragma unroll
            for (int j = 0; j < kSteps[0]; ++j)
                mma_f16(d, a[0] + tap_off<MODE>(tap) + 2 * j, kBoxHi, w + (uint32_t)((tap * WB) >> 4) + 2 * j, kWeightHi, idesc,
                        tap > 0 || j > 0 ? 1u : 0u);
    } else {
        uint32_t row = tap_off<MODE>(MODE == 0 ? 0 : 2);  // the tap row's place in a box
#pragma unroll 1
        for (int ky = 0; ky < 3; ++ky) {
#pragma unroll
            for (int kx = 0; kx < 3; ++kx)
#pragma unroll
                for (int c = 0; c < NCK; ++c)
#pragma unroll
                    for (int j = 0; j < 4; ++j)
                        if (kSteps[c] > 0 ? j < kSteps[c] : j < ks[c])
                            mma_f16(d, a[c] + row + (uint32_t)((MODE == 0 ? kx : 2 - kx) * (128 >> 4) + 2 * j), kBoxHi,
                                    w + (uint32_t)(((c * 9 + kx) * WB) >> 4) + 2 * j, kWeightHi, idesc,
                                    kx > 0 || c > 0 || j > 0 ? 1u : (uint32_t)(ky > 0));
            row += MODE == 0 ? (uint32_t)(ROW_BYTES >> 4) : 0u - (uint32_t)(ROW_BYTES >> 4);
            w += (uint32_t)((3 * WB) >> 4);
        }
    }
}

// The K steps of one or two chunks as compile-time numbers.
template <int MODE, int WB, int... KS>
__device__ __forceinline__ void tile_mmas1(uint32_t d, const uint32_t (&a)[sizeof...(KS) + 1], const int (&ks)[sizeof...(KS) + 1],
                                           uint32_t w, uint32_t idesc) {
    const int k = ks[sizeof...(KS)];
    if (k > 3) tile_mmas<MODE, WB, KS..., 4>(d, a, ks, w, idesc);
    else if (k > 2) tile_mmas<MODE, WB, KS..., 3>(d, a, ks, w, idesc);
    else if (k > 1) tile_mmas<MODE, WB, KS..., 2>(d, a, ks, w, idesc);
    else tile_mmas<MODE, WB, KS..., 1>(d, a, ks, w, idesc);
}
template <int MODE, int WB>
__device__ __forceinline__ void tile_mmas2(uint32_t d, const uint32_t (&a)[2], const int (&ks)[2], uint32_t w, uint32_t idesc) {
    const int k = MODE == 1 ? 4 : ks[0];  // (the data gradient has one input: its first chunk is full)
    if (k > 3) tile_mmas1<MODE, WB, 4>(d, a, ks, w, idesc);
    else if (k > 2) tile_mmas1<MODE, WB, 3>(d, a, ks, w, idesc);
    else if (k > 1) tile_mmas1<MODE, WB, 2>(d, a, ks, w, idesc);
    else tile_mmas1<MODE, WB, 1>(d, a, ks, w, idesc);
}

// MODE 0 (forward): A = [x1 | x2] (C1 + C2 channels), B = Wb as [cout][9][cin], out =
// o1 (Co1 = cout channels, + bias, ReLU).  MODE 1 (data gradient): A = dy (C1 = cout
// channels, C2 = 0, the ReLU derivative applied before), taps mirrored, B = Wt as
// [9][cin][cout], out = [o1 | o2].  NB: output channels of a CTA.  C8: eight input
// channels (forward).
template <int MODE, int RELU, int NB, bool C8>
__global__ void __launch_bounds__(TILE_THREADS, 1)
k_conv_tile(const __grid_constant__ CUtensorMap ta1, const __grid_constant__ CUtensorMap ta2,
            const __grid_constant__ CUtensorMap tb, const float* __restrict__ bias, bf16* __restrict__ o1, int Co1,
            bf16* __restrict__ o2, int Co2, int C1, int C2, int H, int W, int ntx, int nty, int ntiles, int NT,
            TileShape sh, int* err) {
    constexpr uint32_t kCols = NB <= 16 ? 32u : (NB <= 32 ? 64u : (NB <= 64 ? 128u : 256u));
    constexpr int WB = C8 ? NB * 16 : NB * 128;  // weights of one tap and chunk
    constexpr int BOX = C8 ? BOX8_BYTES : BOX_BYTES;
    constexpr uint32_t kIdescT = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(NB >> 3) << 17) | (8u << 24);
    extern __shared__ unsigned char smem_raw[];
    unsigned char* smem = (unsigned char*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    unsigned char* zeros = smem + sh.stages * BOX;  // C8
    unsigned char* wres = zeros + (C8 ? ZERO8_BYTES : 0);
    uint64_t* full = (uint64_t*)(wres + sh.nck * (C8 ? 10 : 9) * WB);
    uint64_t* empty = full + kTileStagesMax;
    uint64_t* acc_full = empty + kTileStagesMax;
    uint64_t* acc_empty = acc_full + ACC;
    uint64_t* b_full = acc_empty + ACC;
    uint32_t* tslot = (uint32_t*)(b_full + 1);
    float* sbias = (float*)(tslot + 2);
    const int tid = threadIdx.x, warp = warp_id(), lane = tid & 31;
    const int cpn = gridDim.x / NT, n0 = (blockIdx.x % NT) * NB, t0 = blockIdx.x / NT;
    const int Nout = Co1 + Co2, S = sh.stages;

    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;\n" ::"r"(saddr(tslot)), "r"(kCols)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n" ::: "memory");
    }
    if (tid == 0) {
        for (int q = 0; q < S; ++q) {
            asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;\n" ::"r"(saddr(full + q)) : "memory");
            asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;\n" ::"r"(saddr(empty + q)) : "memory");
        }
        for (int q = 0; q < ACC; ++q) {
            asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;\n" ::"r"(saddr(acc_full + q)) : "memory");
            asm volatile("mbarrier.init.shared::cta.b64 [%0], 4;\n" ::"r"(saddr(acc_empty + q)) : "memory");
        }
        asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;\n" ::"r"(saddr(b_full)) : "memory");
        asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
    }
    if (C8) {  // tap 9: no activations, no weights
        for (int e = tid; e < ZERO8_BYTES / 16; e += TILE_THREADS) ((uint4*)zeros)[e] = make_uint4(0u, 0u, 0u, 0u);
        for (int e = tid; e < WB / 16; e += TILE_THREADS) ((uint4*)(wres + 9 * WB))[e] = make_uint4(0u, 0u, 0u, 0u);
        asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
    }
    if (MODE == 0 && tid >= 64 && tid - 64 < NB) sbias[tid - 64] = n0 + tid - 64 < Nout ? bias[n0 + tid - 64] : 0.f;
    asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
    const uint32_t tmem = __shfl_sync(0xffffffffu, *tslot, 0);
    bool ok = true;

    if (warp == 0) {
        if (lane == 0) {
            asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;\n" ::"r"(saddr(b_full)),
                         "r"((uint32_t)(sh.nck * 9 * WB))
                         : "memory");
            for (int ck = 0; ck < sh.nck; ++ck) {
                const int c = ck < sh.nck1 ? ck * 64 : C1 + (ck - sh.nck1) * 64;
                for (int tap = 0; tap < 9; ++tap) {
                    const uint32_t dst = saddr(wres + (ck * 9 + tap) * WB);
                    if (MODE == 0) tma_load_3d(dst, &tb, c, tap, n0, saddr(b_full));
                    else tma_load_3d(dst, &tb, c, n0, tap, saddr(b_full));
                }
            }
            int g = 0, st = 0;  // stages filled, across tiles
            uint32_t ph = 1u;   // parity of a stage's last release (none needed in the first round)
            for (int t = t0; t < ntiles && ok; t += cpn) {
                const int img = t / (ntx * nty), r = t - img * ntx * nty, y0 = r / ntx * TH, x0 = r % ntx * TW;
                for (int ck = 0; ck < sh.nck; ++ck, ++g) {
                    if (g >= S && !wait_parity(saddr(empty + st), ph)) {
                        ok = false;
                        break;
                    }
                    const uint32_t bar = saddr(full + st), dst = saddr(smem) + st * BOX;
                    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;\n" ::"r"(bar), "r"((uint32_t)BOX)
                                 : "memory");
                    if (ck < sh.nck1) tma_load_4d(dst, &ta1, ck * 64, x0 - 1, y0 - 1, img, bar);
                    else tma_load_4d(dst, &ta2, (ck - sh.nck1) * 64, x0 - 1, y0 - 1, img, bar);
                    if (++st == S) {
                        st = 0;
                        ph ^= 1u;
                    }
                }
            }
            // copies still in flight land before the CTA leaves (bounded waits)
            wait_parity(saddr(b_full), 0u);
            for (int q = 0; q < S && q < g; ++q) {
                const int gg = g - 1 - q, st = gg % S, use = gg / S;
                wait_parity(saddr(full + st), (uint32_t)(use & 1));
            }
        }
        __syncwarp();
    } else if (warp == 1) {
        // the whole warp in step, an elected lane issues (mma_f16)
        ok = wait_parity_warp(saddr(b_full), 0u);
        asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
        // (stage and accumulator numbers and parities are carried along: a single warp's
        // instructions between the MMAs are on the critical path)
        const uint32_t box0 = desc_lo(saddr(smem)), w0 = desc_lo(saddr(wres)), full0 = saddr(full), empty0 = saddr(empty);
        int st = 0, acc = 0, lt = 0;
        uint32_t ph = 0u, aph = 1u;
        for (int t = t0; t < ntiles && ok; t += cpn, ++lt) {
            if (lt >= ACC && !wait_parity_warp(saddr(acc_empty + acc), aph)) {
                ok = false;
                break;
            }
            const uint32_t d = tmem + (uint32_t)(acc * NB);
            if constexpr (C8) {
                if (!wait_parity_warp(full0 + 8 * st, ph)) ok = false;
                asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
                // K-major without swizzle: core matrices of eight pixels x 16 B; image rows
                // 256 B apart; the step's second tap at the leading offset
                constexpr uint32_t hiA = (256u >> 4) | (1u << 14), hiB = (128u >> 4) | (1u << 14);
                const uint32_t a = (saddr(smem) + (uint32_t)st * BOX) >> 4, b = saddr(wres) >> 4;
                const uint32_t zoff = (saddr(zeros) >> 4) - (a + (544u >> 4));
                if (ok) {
#pragma unroll
                    for (int q = 0; q < 5; ++q) {
                        constexpr int off[10] = {0, 16, 32, 256, 272, 288, 512, 528, 544, 0};
                        const uint32_t lead = q < 4 ? (uint32_t)(off[2 * q + 1] - off[2 * q]) >> 4 : zoff;
                        mma_f16(d, (a + (uint32_t)(off[2 * q] >> 4)) | (lead << 16), hiA,
                                (b + (uint32_t)((2 * q * WB) >> 4)) | ((uint32_t)(WB >> 4) << 16), hiB, kIdescT, q > 0 ? 1u : 0u);
                    }
                }
                mma_commit(empty0 + 8 * st);
                if (++st == S) {
                    st = 0;
                    ph ^= 1u;
                }
            } else {
                // all chunks' boxes of the tile (S >= nck), then tap by tap through the chunks
                int s1 = st;
                uint32_t p1 = ph;
                for (int ck = 0; ck < sh.nck && ok; ++ck) {
                    ok = wait_parity_warp(full0 + 8 * s1, p1);
                    if (++s1 == S) {
                        s1 = 0;
                        p1 ^= 1u;
                    }
                }
                asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
                // (a copy did not arrive: nothing is multiplied, the tile is committed as it is)
                auto go = [&](auto nck) {
                    constexpr int NCK = decltype(nck)::value;
                    uint32_t a[NCK];
                    int ks[NCK];
#pragma unroll
                    for (int c = 0; c < NCK; ++c) {
                        const int left = c == 0 || c < sh.nck1 ? C1 - c * 64 : C2 - (c - sh.nck1) * 64;
                        ks[c] = min(4, (left + 15) / 16);
                        a[c] = box0 + (uint32_t)(c == 0 || st + c < S ? st + c : st + c - S) * (BOX_BYTES >> 4);
                    }
                    if constexpr (NCK == 1) tile_mmas1<MODE, WB>(d, a, ks, w0, kIdescT);
                    else if constexpr (NCK == 2) tile_mmas2<MODE, WB>(d, a, ks, w0, kIdescT);
                    else if constexpr (NCK == 3) tile_mmas<MODE, WB, 0, 0, 0>(d, a, ks, w0, kIdescT);
                    else tile_mmas<MODE, WB, 0, 0, 0, 0>(d, a, ks, w0, kIdescT);
                };
                if (ok) {
                    if (sh.nck == 1) go(std::integral_constant<int, 1>{});
                    else if (sh.nck == 2) go(std::integral_constant<int, 2>{});
                    else if (sh.nck == 3) go(std::integral_constant<int, 3>{});
                    else go(std::integral_constant<int, 4>{});
                }
                for (int ck = 0; ck < sh.nck; ++ck) mma_commit(empty0 + 8 * (st + ck < S ? st + ck : st + ck - S));
                st = s1;
                ph = p1;
            }
            // committed even after a failed wait, so the epilogue's wait ends
            mma_commit(saddr(acc_full + acc));
            if (++acc == ACC) {
                acc = 0;
                aph ^= 1u;
            }
        }
        __syncwarp();
    } else {
        const int quarter = warp & 3, m = quarter * 32 + lane;
        int lt = 0;
        for (int t = t0; t < ntiles; t += cpn, ++lt) {
            const int acc = lt % ACC, ause = lt / ACC;
            const bool got = wait_parity(saddr(acc_full + acc), (uint32_t)(ause & 1));
            asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
            if (!got) {
                ok = false;
                break;
            }
            const int img = t / (ntx * nty), r0 = t - img * ntx * nty;
            const int y = r0 / ntx * TH + (m >> 3), x = r0 % ntx * TW + (m & 7);
            const bool in = y < H && x < W;
            const size_t p = ((size_t)img * H + y) * W + x;
#pragma unroll
            for (int c = 0; c < NB; c += 16) {
                uint32_t r[16];
                asm volatile(
                    "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];\n"
                    : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
                      "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
                    : "r"(tmem + ((uint32_t)(quarter * 32) << 16) + (uint32_t)(acc * NB + c))
                    : "memory");
                asm volatile("tcgen05.wait::ld.sync.aligned;\n" ::: "memory");
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    const int col = n0 + c + 8 * h;  // eight channels, all in o1 or all in o2
                    uint4 v;
                    __nv_bfloat162* w2 = (__nv_bfloat162*)&v;
#pragma unroll
                    for (int q = 0; q < 4; ++q) {
                        float v0 = __uint_as_float(r[8 * h + 2 * q]), v1 = __uint_as_float(r[8 * h + 2 * q + 1]);
                        if (MODE == 0) {
                            v0 += sbias[c + 8 * h + 2 * q];
                            v1 += sbias[c + 8 * h + 2 * q + 1];
                            if (RELU) {
                                v0 = fmaxf(v0, 0.f);
                                v1 = fmaxf(v1, 0.f);
                            }
                        }
                        w2[q] = __floats2bfloat162_rn(v0, v1);
                    }
                    if (in && col < Nout) *(uint4*)(col < Co1 ? o1 + p * Co1 + col : o2 + p * Co2 + (col - Co1)) = v;
                }
            }
            asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
            __syncwarp();
            if (lane == 0)
                asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];\n" ::"r"(saddr(acc_empty + acc)) : "memory");
        }
    }
    if (!ok) atomicExch(err, 1);
    asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
    __syncthreads();
    if (warp == 0)
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;\n" ::"r"(tmem), "r"(kCols) : "memory");
}

// ---------------------------------------------------------------------------
// Weight gradient, as k_conv_wgrad_tma (nn_tc.cu: M = two taps x 64 input channels, N =
// output channels, K = pixels, MN-major boxes of 64 pixels, split-K), with 8 x 8-pixel
// boxes, so that images of any size are covered, and channels beyond the counts filled with
// zeros and not stored.  Pixels of a box outside the image count as zero in both operands:
// the copy engine fills dy with zeros there, and the rows of x, which its shift may take from
// inside the image, are cleared before the MMAs (0 times an infinite x is NaN).  NB: output
// channels of a CTA (an MMA's N).
// ---------------------------------------------------------------------------
constexpr int WT_BOX = 64 * 128;        // 64 pixels x 64 channels
constexpr int WT_STAGE = 3 * WT_BOX;    // two tap boxes of x, dy
constexpr int WT_STAGES = 3, WT_THREADS = 128;
// accumulators that take the K steps in turn and are added at the end: the FP32 rounding
// of a sum grows with its length (error of dW against 64 bits, 18 images, 8 -> 32 channels
// at 120 x 128: 2.6e-6 with one accumulator, 2.6e-7 with eight, mma.sync kernel 4.8e-7; 32
// -> 32 at 128^2: 2.9e-7 with eight, mma.sync kernel 1.2e-6)
template <int NB> constexpr int kWtAcc = NB <= 32 ? 8 : 4;  // at most 256 TMEM columns: two CTAs per SM
constexpr int WT_SMEM = WT_STAGES * WT_STAGE + 1024 + (2 * WT_STAGES + 2) * 8;

template <int NB>
__global__ void __launch_bounds__(WT_THREADS)
k_conv_wgrad_tile(const __grid_constant__ CUtensorMap tx1, const __grid_constant__ CUtensorMap tx2,
                  const __grid_constant__ CUtensorMap tdy, float* __restrict__ ws, int C1, int C2, int Cout, int H, int W,
                  int nck1, int nck, int ntx, int nty, int nboxes, int chunk, int* err) {
    constexpr int ACCS = kWtAcc<NB>;
    constexpr uint32_t kCols = ACCS * NB;
    constexpr uint32_t kIdescT = (1u << 4) | (1u << 7) | (1u << 10) | (1u << 15) | (1u << 16) |
                                 ((uint32_t)(NB >> 3) << 17) | (8u << 24);
    extern __shared__ unsigned char smem_raw[];
    unsigned char* smem = (unsigned char*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    uint64_t* full = (uint64_t*)(smem + WT_STAGES * WT_STAGE);
    uint64_t* empty = full + WT_STAGES;
    uint64_t* done = empty + WT_STAGES;
    uint32_t* tslot = (uint32_t*)(done + 1);
    const int tid = threadIdx.x, warp = warp_id(), lane = tid & 31;
    const int Cin = C1 + C2, nco = (Cout + NB - 1) / NB;
    int t = blockIdx.x;
    const int n0 = t % nco * NB;
    t /= nco;
    const int ck = t % nck, g = t / nck;  // input-channel chunk, tap pair
    const int tap0 = 2 * g, tap1 = g < 4 ? 2 * g + 1 : 8;
    const int q0 = blockIdx.y * chunk, q1 = min(nboxes, q0 + chunk), nk = q1 > q0 ? q1 - q0 : 0;
    const bool first = ck < nck1;
    const int c = first ? ck * 64 : (ck - nck1) * 64;              // in its input
    const int valid = min(64, (first ? C1 : C2) - c), c_out = first ? c : C1 + c;

    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;\n" ::"r"(saddr(tslot)), "r"(kCols)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n" ::: "memory");
    }
    if (tid == 0) {
        for (int q = 0; q < WT_STAGES; ++q) {
            asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;\n" ::"r"(saddr(full + q)) : "memory");
            asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;\n" ::"r"(saddr(empty + q)) : "memory");
        }
        asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;\n" ::"r"(saddr(done)) : "memory");
        asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
    const uint32_t tmem = *tslot;
    bool ok = true;
    if (nk > 0) {
        if (warp == 0) {
            if (lane == 0) {
                const int dy0 = tap0 / 3 - 1, dx0 = tap0 % 3 - 1, dy1 = tap1 / 3 - 1, dx1 = tap1 % 3 - 1;
                const CUtensorMap* xm = first ? &tx1 : &tx2;
                for (int kc = 0; kc < nk; ++kc) {
                    const int st = kc % WT_STAGES, use = kc / WT_STAGES;
                    if (use > 0 && !wait_parity(saddr(empty + st), (uint32_t)((use + 1) & 1))) {
                        ok = false;
                        break;
                    }
                    const int q = q0 + kc, img = q / (ntx * nty), r = q - img * ntx * nty, y0 = r / ntx * 8, x0 = r % ntx * 8;
                    const uint32_t dst = saddr(smem + st * WT_STAGE);
                    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;\n" ::"r"(saddr(full + st)),
                                 "r"((uint32_t)WT_STAGE)
                                 : "memory");
                    tma_load_4d(dst, xm, c, x0 + dx0, y0 + dy0, img, saddr(full + st));
                    tma_load_4d(dst + WT_BOX, xm, c, x0 + dx1, y0 + dy1, img, saddr(full + st));
                    tma_load_4d(dst + 2 * WT_BOX, &tdy, n0, x0, y0, img, saddr(full + st));
                }
            }
            __syncwarp();
        } else if (warp == 1) {
            const bool ragged = (H & 7) != 0 || (W & 7) != 0;
            int bx = q0 % ntx, by = q0 / ntx % nty;  // the box's place in its image
            for (int kc = 0; kc < nk; ++kc) {
                const int st = kc % WT_STAGES, use = kc / WT_STAGES;
                if (!wait_parity_warp(saddr(full + st), (uint32_t)(use & 1))) {
                    ok = false;
                    break;
                }
                if (ragged) {
                    const int y1 = H - by * 8, x1 = W - bx * 8;  // rows and columns of the box inside the image
                    if (y1 < 8 || x1 < 8) {                      // (uniform)
                        for (int p = lane; p < 128; p += 32) {   // 64 pixels of each tap, a row of 128 bytes each
                            if ((p >> 3 & 7) < y1 && (p & 7) < x1) continue;
                            uint4* row = (uint4*)(smem + st * WT_STAGE + p * 128);
#pragma unroll
                            for (int v = 0; v < 8; ++v) row[v] = make_uint4(0u, 0u, 0u, 0u);
                        }
                        asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
                        __syncwarp();
                    }
                    if (++bx == ntx) {
                        bx = 0;
                        if (++by == nty) by = 0;
                    }
                }
                asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
                const uint32_t a = desc_lo_mn(saddr(smem + st * WT_STAGE), WT_BOX), b = a + ((2 * WT_BOX) >> 4);
#pragma unroll
                for (int j = 0; j < 4; ++j)
                    mma_f16(tmem + (uint32_t)((kc % (ACCS / 4) * 4 + j) * NB), a + 128 * j, kWeightHi, b + 128 * j, kWeightHi,
                            kIdescT, kc >= ACCS / 4 ? 1u : 0u);
                mma_commit(saddr(empty + st));
            }
            mma_commit(saddr(done));
            __syncwarp();
        }
        if (!wait_parity(saddr(done), 0u)) ok = false;
        asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
    }
    if (__syncthreads_or(ok ? 0 : 1)) ok = false;
    // TMEM lane m = warp * 32 + lane: tap (m < 64 ? tap0 : tap1), input channel c + m % 64
    const int m = warp * 32 + lane, tap = m < 64 ? tap0 : tap1;
    const bool store = (m < 64 || g < 4) && (m & 63) < valid;
    float* out = ws + (size_t)blockIdx.y * Cout * 9 * Cin + (size_t)tap * Cin + c_out + (m & 63);
    const int accs = min(4 * nk, ACCS);
#pragma unroll
    for (int col = 0; col < NB; col += 16) {
        float v[16];
#pragma unroll
        for (int q = 0; q < 16; ++q) v[q] = 0.f;
        for (int k = 0; k < accs; ++k) {
            uint32_t r[16];
            asm volatile(
                "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];\n"
                : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
                  "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
                : "r"(tmem + ((uint32_t)(warp * 32) << 16) + (uint32_t)(k * NB + col))
                : "memory");
            asm volatile("tcgen05.wait::ld.sync.aligned;\n" ::: "memory");
#pragma unroll
            for (int q = 0; q < 16; ++q) v[q] += __uint_as_float(r[q]);
        }
        if (store) {
#pragma unroll
            for (int q = 0; q < 16; ++q)
                if (n0 + col + q < Cout) out[(size_t)(n0 + col + q) * 9 * Cin] = ok ? v[q] : __int_as_float(0x7fc00000);
        }
    }
    if (!ok && tid == 0) atomicExch(err, 1);
    asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
    __syncthreads();
    if (warp == 0)
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;\n" ::"r"(tmem), "r"(kCols) : "memory");
}

// ---------------------------------------------------------------------------
// host side
// ---------------------------------------------------------------------------

static bool map4(CUtensorMap* m, const void* base, int c, int n, int h, int w, int bw, int bh, int bc = 64) {
    PFN_cuTensorMapEncodeTiled_v12000 enc = tmap_encoder();
    if (!enc) return false;
    cuuint64_t dims[4] = {(cuuint64_t)c, (cuuint64_t)w, (cuuint64_t)h, (cuuint64_t)n};
    cuuint64_t strides[3] = {(cuuint64_t)c * 2, (cuuint64_t)w * c * 2, (cuuint64_t)h * w * c * 2};
    cuuint32_t box[4] = {(cuuint32_t)bc, (cuuint32_t)bw, (cuuint32_t)bh, 1u};
    cuuint32_t es[4] = {1u, 1u, 1u, 1u};
    return enc(m, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 4, const_cast<void*>(base), dims, strides, box, es,
               CU_TENSOR_MAP_INTERLEAVE_NONE, bc == 64 ? CU_TENSOR_MAP_SWIZZLE_128B : CU_TENSOR_MAP_SWIZZLE_NONE,
               CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

static bool map3(CUtensorMap* m, const void* base, long long d0, long long d1, long long d2, int b1, int b2, int b0 = 64) {
    PFN_cuTensorMapEncodeTiled_v12000 enc = tmap_encoder();
    if (!enc) return false;
    cuuint64_t dims[3] = {(cuuint64_t)d0, (cuuint64_t)d1, (cuuint64_t)d2};
    cuuint64_t strides[2] = {(cuuint64_t)d0 * 2, (cuuint64_t)(d0 * d1) * 2};
    cuuint32_t box[3] = {(cuuint32_t)b0, (cuuint32_t)b1, (cuuint32_t)b2};
    cuuint32_t es[3] = {1u, 1u, 1u};
    return enc(m, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, const_cast<void*>(base), dims, strides, box, es,
               CU_TENSOR_MAP_INTERLEAVE_NONE, b0 == 64 ? CU_TENSOR_MAP_SWIZZLE_128B : CU_TENSOR_MAP_SWIZZLE_NONE,
               CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

static int chunks(int c) { return (c + 63) / 64; }

static int tile_smem(int nck, int stages, int nb, bool c8) {
    const int data = c8 ? stages * BOX8_BYTES + ZERO8_BYTES + 10 * nb * 16 : stages * BOX_BYTES + nck * 9 * nb * 128;
    return data + (2 * kTileStagesMax + 2 * ACC + 2) * 8 + nb * 4 + 1024;
}

// Output channels of a CTA: all of them where their weights fit beside two operand
// stages (the activations are then loaded once), else the widest of 64, 32 and 16 that
// leaves room for a whole tile's boxes; 0: none does (more than 256 input channels).
static int tile_nb(int nck, int nout) {
    const int all[] = {16, 32, 64, 96, 128}, part[] = {64, 32, 16};
    const int need = nck < 2 ? 2 : nck;
    for (int nb : all)
        if (nb >= nout && tile_smem(nck, need, nb, false) <= SMEM_MAX) return nb;
    for (int nb : part)
        if (need <= kTileStagesMax && tile_smem(nck, need, nb, false) <= SMEM_MAX) return nb;
    return 0;
}

static int sm_count() {
    int dev = 0, sms = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    return sms > 0 ? sms : 152;
}

template <int MODE, int RELU, int NB, bool C8>
static int launch_tile(const CUtensorMap& t1, const CUtensorMap& t2, const CUtensorMap& tb, const float* bias, void* o1,
                       int co1, void* o2, int co2, int c1, int c2, int n, int h, int w, int* err, cudaStream_t s) {
    static cudaError_t attr =
        cudaFuncSetAttribute(k_conv_tile<MODE, RELU, NB, C8>, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM_MAX);
    if (attr != cudaSuccess) return 0;
    TileShape sh;
    sh.nck1 = chunks(c1);
    sh.nck = sh.nck1 + chunks(c2);
    sh.stages = kTileStagesMax;
    while (tile_smem(sh.nck, sh.stages, NB, C8) > SMEM_MAX) --sh.stages;
    if (sh.stages < sh.nck) return 0;
    sh.smem = tile_smem(sh.nck, sh.stages, NB, C8);
    const int ntx = (w + TW - 1) / TW, nty = (h + TH - 1) / TH, NT = (co1 + co2 + NB - 1) / NB;
    const long long ntiles = (long long)n * ntx * nty;
    // one CTA per SM: its stages and weights fill the shared memory (eight channels: two)
    long long cpn = (long long)sm_count() * (C8 ? 2 : 1) / NT;
    cpn = cpn < 1 ? 1 : (cpn > ntiles ? ntiles : cpn);
    k_conv_tile<MODE, RELU, NB, C8><<<(unsigned)(NT * cpn), TILE_THREADS, sh.smem, s>>>(
        t1, t2, tb, bias, (bf16*)o1, co1, (bf16*)o2, co2, c1, c2, h, w, ntx, nty, (int)ntiles, NT, sh, err);
    return 1;
}

template <int MODE, int RELU>
static int launch_tile_nb(int nb, const CUtensorMap& t1, const CUtensorMap& t2, const CUtensorMap& tb, const float* bias,
                          void* o1, int co1, void* o2, int co2, int c1, int c2, int n, int h, int w, int* err,
                          cudaStream_t s) {
    switch (nb) {
        case 16: return launch_tile<MODE, RELU, 16, false>(t1, t2, tb, bias, o1, co1, o2, co2, c1, c2, n, h, w, err, s);
        case 32: return launch_tile<MODE, RELU, 32, false>(t1, t2, tb, bias, o1, co1, o2, co2, c1, c2, n, h, w, err, s);
        case 64: return launch_tile<MODE, RELU, 64, false>(t1, t2, tb, bias, o1, co1, o2, co2, c1, c2, n, h, w, err, s);
        case 96: return launch_tile<MODE, RELU, 96, false>(t1, t2, tb, bias, o1, co1, o2, co2, c1, c2, n, h, w, err, s);
        case 128: return launch_tile<MODE, RELU, 128, false>(t1, t2, tb, bias, o1, co1, o2, co2, c1, c2, n, h, w, err, s);
    }
    return 0;
}

}  // namespace glnn_tc

using namespace glnn_tc;

// 1: launched; 0: not taken (the caller uses the thread-gather kernel)
int glnn_tile_fwd(const void* x1, int c1, const void* x2, int c2, const void* wb, const float* bias, void* y, int n, int h,
                  int w, int cout, int relu, int* err, cudaStream_t s) {
    if (c1 == 8 && c2 == 0) {  // the CTA's output channels in one piece
        CUtensorMap t1, tb;
        const int nb = cout <= 32 ? 32 : 64;
        if (!map4(&t1, x1, 8, n, h, w, BOXW, BOXH, 8) || !map3(&tb, wb, 8, 9, cout, 1, nb, 8)) return 0;
        if (nb == 32)
            return relu ? launch_tile<0, 1, 32, true>(t1, t1, tb, bias, y, cout, nullptr, 0, 8, 0, n, h, w, err, s)
                        : launch_tile<0, 0, 32, true>(t1, t1, tb, bias, y, cout, nullptr, 0, 8, 0, n, h, w, err, s);
        return relu ? launch_tile<0, 1, 64, true>(t1, t1, tb, bias, y, cout, nullptr, 0, 8, 0, n, h, w, err, s)
                    : launch_tile<0, 0, 64, true>(t1, t1, tb, bias, y, cout, nullptr, 0, 8, 0, n, h, w, err, s);
    }
    // K steps of 16 channels as the thread-gather kernel takes them: none across taps or inputs
    const int nb = tile_nb(chunks(c1) + chunks(c2), cout);
    if (!nb || c1 % 16 || c2 % 16) return 0;
    CUtensorMap t1, t2, tb;
    if (!map4(&t1, x1, c1, n, h, w, BOXW, BOXH) || !map3(&tb, wb, c1 + c2, 9, cout, 1, nb)) return 0;
    t2 = t1;
    if (c2 > 0 && !map4(&t2, x2, c2, n, h, w, BOXW, BOXH)) return 0;
    return relu ? launch_tile_nb<0, 1>(nb, t1, t2, tb, bias, y, cout, nullptr, 0, c1, c2, n, h, w, err, s)
                : launch_tile_nb<0, 0>(nb, t1, t2, tb, bias, y, cout, nullptr, 0, c1, c2, n, h, w, err, s);
}

// dy with the ReLU derivative already applied
int glnn_tile_bwd_data(const void* dy, const void* wt, void* dx1, int c1, void* dx2, int c2, int n, int h, int w, int cout,
                       int* err, cudaStream_t s) {
    const int nb = tile_nb(chunks(cout), c1 + c2);
    if (!nb) return 0;
    CUtensorMap ta, tb;
    if (!map4(&ta, dy, cout, n, h, w, BOXW, BOXH) || !map3(&tb, wt, cout, c1 + c2, 9, nb, 1)) return 0;
    return launch_tile_nb<1, 0>(nb, ta, ta, tb, nullptr, dx1, c1, dx2, c2, cout, 0, n, h, w, err, s);
}

// split-K plan: about two CTAs per SM in all
static void wgrad_tile_plan(int n, int h, int w, int c1, int c2, int cout, int* nz, int* chunk, int* nb, int* tiles) {
    *nb = cout <= 16 ? 16 : (cout <= 32 ? 32 : 64);
    *tiles = 5 * (chunks(c1) + chunks(c2)) * ((cout + *nb - 1) / *nb);
    const long long boxes = (long long)n * ((h + 7) / 8) * ((w + 7) / 8);
    long long z = (2 * 152 + *tiles - 1) / *tiles;
    z = z < 1 ? 1 : (z > boxes ? boxes : z);
    const long long per = (boxes + z - 1) / z;
    *chunk = (int)per;
    *nz = (int)((boxes + per - 1) / per);
}

// most splits that the tile kernel uses for any grouping of the input channels
int glnn_tile_wgrad_splits(int n, int h, int w, int cin, int cout) {
    int nz = 0, chunk = 0, nb = 0, tiles = 0;
    wgrad_tile_plan(n, h, w, cin, 0, cout, &nz, &chunk, &nb, &tiles);
    return nz;
}

int glnn_tile_wgrad(const void* dy, const void* x1, int c1, const void* x2, int c2, float* ws, int n, int h, int w,
                    int cout, int* nz, int* err, cudaStream_t s) {
    int chunk = 0, nb = 0, tiles = 0;
    wgrad_tile_plan(n, h, w, c1, c2, cout, nz, &chunk, &nb, &tiles);
    CUtensorMap t1, t2, td;
    if (!map4(&t1, x1, c1, n, h, w, 8, 8) || !map4(&td, dy, cout, n, h, w, 8, 8)) return 0;
    t2 = t1;
    if (c2 > 0 && !map4(&t2, x2, c2, n, h, w, 8, 8)) return 0;
    const int ntx = (w + 7) / 8, nty = (h + 7) / 8, nck1 = chunks(c1), nck = nck1 + chunks(c2);
    const dim3 grid((unsigned)tiles, (unsigned)*nz);
    static const bool ready =
        cudaFuncSetAttribute(k_conv_wgrad_tile<16>, cudaFuncAttributeMaxDynamicSharedMemorySize, WT_SMEM) == cudaSuccess &&
        cudaFuncSetAttribute(k_conv_wgrad_tile<32>, cudaFuncAttributeMaxDynamicSharedMemorySize, WT_SMEM) == cudaSuccess &&
        cudaFuncSetAttribute(k_conv_wgrad_tile<64>, cudaFuncAttributeMaxDynamicSharedMemorySize, WT_SMEM) == cudaSuccess;
    if (!ready) return 0;
    auto go = [&](auto kernel) {
        kernel<<<grid, WT_THREADS, WT_SMEM, s>>>(t1, t2, td, ws, c1, c2, cout, h, w, nck1, nck, ntx, nty, n * ntx * nty,
                                                   chunk, err);
        return 1;
    };
    return nb == 16 ? go(k_conv_wgrad_tile<16>) : (nb == 32 ? go(k_conv_wgrad_tile<32>) : go(k_conv_wgrad_tile<64>));
}
