// Node arithmetic of the TDGL Jacobi sweeps, shared by the sweep kernels of td.cu, the
// cooperative loops of tdl.cu and the resident time loop of tdr.cu, so that a
// node gets the same operations in the same order on every path.  Fused multiply-adds
// are written out (and mul_rn keeps other products unfused): left to the compiler, the
// choice differs between kernels.
#pragma once

#include "glgpu_common.cuh"

namespace glgpu {

// The backward-Euler Jacobi update of one node (svirl/cuda/td.h:4-133 with the
// Winecki-Adams link weights of td.h:159-163, coded as bits of cd: 0 left,
// 1 right, 2 lower, 3 upper link), in two parts.  The diagonal depends only on
// the right-hand side (with the Langevin term, rq), the linear coefficient and
// the link weights, which are fixed during a Jacobi loop, so its reciprocal is
// formed once per node and launch (psi_diag_inv) and each sweep only forms the
// neighbour sums (psi_node).  A node with neither a left nor a right link gets 0.
// The link table holds U scaled by dt/dx^2 (x links) or dt/dy^2 (y links), and
// 0 on links of weight 0, so the neighbour sum is one FMA chain per component
// with no branch per link.
template <typename T>
__device__ __forceinline__ T psi_diag_inv(C2<T> rq, T eps, unsigned cd, T dt, T idx2, T idy2) {
    const T a2 = fma(rq.x, rq.x, mul_rn<T>(rq.y, rq.y));
    T links;
    if constexpr (sizeof(T) == 8) {
        // FP64: the link-count terms by selects, keeping conversions off the FP64 pipe
        const unsigned nx = (cd & 1u) + ((cd >> 1) & 1u), ny = ((cd >> 2) & 1u) + ((cd >> 3) & 1u);
        const T cx = nx == 0u ? T(0) : (nx == 1u ? idx2 : idx2 + idx2);
        const T cy = ny == 0u ? T(0) : (ny == 1u ? idy2 : idy2 + idy2);
        links = cx + cy;
    } else {
        const bool rm0 = cd & 1u, rp0 = cd & 2u, r0m = cd & 4u, r0p = cd & 8u;
        const T wx = T(rm0) + T(rp0), wy = T(r0m) + T(r0p);
        links = fma(idx2, wx, mul_rn<T>(idy2, wy));
    }
    return T(1) / fma(dt, (a2 - eps) + links, T(1));
}

// x + c (u - 1/2): the Langevin term (svirl/cuda/td.h:147-151,451-454)
template <typename T> __device__ __forceinline__ T add_noise(T x, T c, T u) { return fma(c, u - T(0.5), x); }

// rq + conj(ua_left) p_left + ua p_right + conj(ub_down) p_prev + ub p_next as one
// FMA chain per component, the link factors already scaled; p_next, the row the
// previous sweep produced last, enters at the end of the chain.
template <typename T>
__device__ __forceinline__ C2<T> psi_node(C2<T> p_left, C2<T> p_right, C2<T> p_prev, C2<T> p_next, C2<T> ua_left,
                                          C2<T> ua, C2<T> ub_down, C2<T> ub, C2<T> rq, T inv, unsigned cd) {
    const C2<T> z = cmk<T>(T(0), T(0));
    C2<T> out = z;
    T ax = fma(ua_left.x, p_left.x, rq.x);
    ax = fma(ua_left.y, p_left.y, ax);
    ax = fma(ua.x, p_right.x, ax);
    ax = fma(-ua.y, p_right.y, ax);
    T ay = fma(ua_left.x, p_left.y, rq.y);
    ay = fma(-ua_left.y, p_left.x, ay);
    ay = fma(ua.x, p_right.y, ay);
    ay = fma(ua.y, p_right.x, ay);
    ax = fma(ub_down.x, p_prev.x, ax);
    ax = fma(ub_down.y, p_prev.y, ax);
    ax = fma(ub.x, p_next.x, ax);
    ax = fma(-ub.y, p_next.y, ax);
    ay = fma(ub_down.x, p_prev.y, ay);
    ay = fma(-ub_down.y, p_prev.x, ay);
    ay = fma(ub.x, p_next.y, ay);
    ay = fma(ub.y, p_next.x, ay);
    const T vx = ax * inv, vy = ay * inv;
    if (cd & 3u) out = cmk<T>(vx, vy);
    return out;
}

// Neighbour terms of the A update of an x link / a y link that starts at a node
// (svirl/cuda/td.h:310-463): values of links outside the domain are passed as 0.
// x link: the x links below and above, the y links that start below (at this node's
// column and the next) and at the link; y link: likewise to the left and right.
// FP32 sums each side by itself: which sweep meets the absolute stop rule hangs on the
// rounding of these sums (|A| reaches H L, the rule is 1e-6), so their order is part of
// the results.  FP64 takes the fewest operations on its pipe.
template <typename T>
__device__ __forceinline__ T A_nbs_x(T idy2, T idxy, T a_dn, T a_up, T b_dn0, T b_dn1, T b0, T b1) {
    if constexpr (sizeof(T) == 8) return fma(idxy, (b_dn1 - b_dn0) + (b0 - b1), mul_rn<T>(idy2, a_dn + a_up));
    else return fma(idxy, b_dn1, fma(idy2, a_dn, -mul_rn<T>(idxy, b_dn0))) + fma(-idxy, b1, fma(idy2, a_up, mul_rn<T>(idxy, b0)));
}
template <typename T>
__device__ __forceinline__ T A_nbs_y(T idx2, T idxy, T b_lt, T b_rt, T a_lt0, T a_lt1, T a0, T a1) {
    if constexpr (sizeof(T) == 8) return fma(idxy, (a_lt1 - a_lt0) + (a0 - a1), mul_rn<T>(idx2, b_lt + b_rt));
    else return fma(idxy, a_lt1, fma(idx2, b_lt, -mul_rn<T>(idxy, a_lt0))) + fma(-idxy, a1, fma(idx2, b_rt, mul_rn<T>(idxy, a0)));
}
// The A^(0) part of an FP32 update (k_A_loop_f32): dt rho k2 (dd nbs(A^(0)) - 2 d^-2 A^(0)).
template <typename T> __device__ __forceinline__ T A_base(T dt_rho_k2, T dd, T nbs, T id2, T a0) {
    return mul_rn<T>(dt_rho_k2, fma(dd, nbs, -mul_rn<T>(T(2) * id2, a0)));
}
// js + field term of a link times dt rho, added to `first` (FP64: the right-hand side
// with its noise; FP32: the noise).
template <typename T> __device__ __forceinline__ T A_fixed(T first, T dt_rho, T jl, T rh) { return fma(dt_rho, jl + rh, first); }

// num / den with rden = 1 / den, den in [1, 2) or a few times that.  FP32 multiplies.
// FP64: one correction of num * rden by its remainder (Markstein 1990: the correctly
// rounded quotient from a correctly rounded reciprocal), three FP64 instructions
// instead of a division's dozen; infinities and NaN pass through.  On 2e8 random operands
// the division's bits, but for quotients below 1e-290 (a subnormal remainder) and the sign
// of a zero.
__device__ __forceinline__ float div_by(float num, float, float rden) { return num * rden; }
__device__ __forceinline__ double div_by(double num, double den, double rden) {
    const double q = num * rden;
    const double c = fma(fma(-q, den, num), rden, q);
    return (__double2hiint(q) & 0x7ff00000) == 0x7ff00000 ? q : c;
}

}  // namespace glgpu
