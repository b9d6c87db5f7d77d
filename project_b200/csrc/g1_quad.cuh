// XYZZ points spread over the four lanes of an aligned quad: lane 0 holds X, lane 1 Y, lane 2 ZZ,
// lane 3 ZZZ.  The fourteen multiplications of an addition form four layers of independent ones, and
// a multiplication costs a warp the same whether one lane or all of them make it, so an addition
// takes the time of four multiplications instead of fourteen (a doubling three instead of nine).
// For sums that a whole call waits for: the few dozen points of a commitment, the tail of an MSM.
#pragma once

#include "g1.cuh"
#include "inverse.cuh"

namespace gzk
{
#if defined(__CUDACC__)
    __device__ __forceinline__ Fp shfl_fp(const Fp& v, int src_lane)
    {
        Fp o;
#pragma unroll
        for (int i = 0; i < FpCfg::N; ++i) o.l[i] = __shfl_sync(0xffffffffu, v.l[i], src_lane);
        return o;
    }
    __device__ __forceinline__ Fp shfl_xor_fp(const Fp& v, int mask)
    {
        Fp o;
#pragma unroll
        for (int i = 0; i < FpCfg::N; ++i) o.l[i] = __shfl_xor_sync(0xffffffffu, v.l[i], mask);
        return o;
    }
    __device__ __forceinline__ Fp select_fp(bool first, const Fp& a, const Fp& b)
    {
        Fp o;
#pragma unroll
        for (int i = 0; i < FpCfg::N; ++i) o.l[i] = first ? a.l[i] : b.l[i];
        return o;
    }
    // One multiplication for all callers: inlined twenty times over, a kernel that runs once per call would spend
    // its time fetching instructions.
    static __device__ __noinline__ Fp quad_mul(const Fp a, const Fp b) { return mul(a, b); }

    // The component of this lane of an affine point, or of the point at infinity (0, 0) where it is that or `take`
    // is false; called by whole warps.
    __device__ __forceinline__ Fp quad_from_affine(const G1Affine* p, bool take)
    {
        const int lane = threadIdx.x & 31, quad = lane & ~3, role = lane & 3;
        Fp c = Fp::zero();
        if (take && role < 2) c = load_fp(role == 0 ? &p->x : &p->y);
        const uint32_t zero = __ballot_sync(0xffffffffu, c.is_zero()) >> quad;
        return role >= 2 && (zero & 3u) != 3u ? Fp::one() : c;
    }

    // p + q and its doubling as one lane computes them (operands that coincide; the sum that vanishes)
    static __device__ __noinline__ Fp quad_add_special(const Fp p, const Fp q)
    {
        const int lane = threadIdx.x & 31, quad = lane & ~3, role = lane & 3;
        G1Xyzz a, b;
        a.X = shfl_fp(p, quad);
        a.Y = shfl_fp(p, quad + 1);
        a.ZZ = shfl_fp(p, quad + 2);
        a.ZZZ = shfl_fp(p, quad + 3);
        b.X = shfl_fp(q, quad);
        b.Y = shfl_fp(q, quad + 1);
        b.ZZ = shfl_fp(q, quad + 2);
        b.ZZZ = shfl_fp(q, quad + 3);
        const G1Xyzz s = g1_add(a, b);
        return role == 0 ? s.X : role == 1 ? s.Y : role == 2 ? s.ZZ : s.ZZZ;
    }

    // p + q, any operands; called by whole warps.
    __device__ __forceinline__ Fp quad_add(const Fp& p, const Fp& q)
    {
        const int lane = threadIdx.x & 31, quad = lane & ~3, role = lane & 3;
        // layer 1: U1 = X1 ZZ2 | S1 = Y1 ZZZ2 | U2 = ZZ1 X2 | S2 = ZZZ1 Y2
        const Fp m = quad_mul(p, shfl_xor_fp(q, 2));
        const Fp o = shfl_xor_fp(m, 2);
        // lanes 0, 2: P = U2 - U1, lanes 1, 3: R = S2 - S1
        const Fp d = sub(select_fp(role < 2, o, m), select_fp(role < 2, m, o));
        const uint32_t zero_p = __ballot_sync(0xffffffffu, p.is_zero()) >> quad, zero_q = __ballot_sync(0xffffffffu, q.is_zero()) >> quad;
        const uint32_t zero_d = __ballot_sync(0xffffffffu, d.is_zero()) >> quad;
        const bool p_infinity = (zero_p & 4u) != 0, q_infinity = (zero_q & 4u) != 0, same_x = (zero_d & 1u) != 0;
        // layer 2: PP = P^2 | R^2 | ZZ1 ZZ2 | ZZZ1 ZZZ2
        const Fp s = quad_mul(select_fp(role < 2, d, p), select_fp(role < 2, d, q));
        // layer 3: PPP = P PP | Q = U1 PP | ZZ3 = ZZ1 ZZ2 PP
        const Fp pp = shfl_fp(s, quad), u1 = shfl_fp(m, quad);
        const Fp t = quad_mul(role == 0 ? d : role == 1 ? u1 : s, pp);
        // layer 4: S1 PPP | R (Q - X3) | - | ZZZ3 = ZZZ1 ZZZ2 PPP, with X3 = R^2 - PPP - 2 Q formed by lane 1
        const Fp ppp = shfl_fp(t, quad), s1 = shfl_fp(m, quad + 1);
        const Fp x3 = sub(sub(s, ppp), add(t, t));
        const Fp f = quad_mul(role == 0 ? s1 : role == 1 ? d : s, role == 1 ? sub(t, x3) : ppp);
        const Fp x3_lane0 = shfl_fp(x3, quad + 1), s1_ppp = shfl_fp(f, quad);
        Fp sum = role == 0 ? x3_lane0 : role == 1 ? sub(f, s1_ppp) : role == 2 ? t : f;
        const bool special = same_x && !p_infinity && !q_infinity;
        if (__any_sync(0xffffffffu, special)) sum = select_fp(special, quad_add_special(p, q), sum);
        return select_fp(q_infinity, p, select_fp(p_infinity, q, sum));
    }

    // 2 p; called by whole warps.  (The curve has no point of order two, and ZZ = 0 stays ZZ = 0.)
    __device__ __forceinline__ Fp quad_double(const Fp& p)
    {
        const int lane = threadIdx.x & 31, quad = lane & ~3, role = lane & 3;
        // layer 1: X^2 | V = U^2 with U = 2 Y
        const Fp twice = add(p, p);
        const Fp s = quad_mul(role == 1 ? twice : p, role == 1 ? twice : p);
        // layer 2: S = X V | W = U V | ZZ V | M^2 with M = 3 X^2
        const Fp v = shfl_fp(s, quad + 1), xx = shfl_fp(s, quad);
        const Fp m = add(add(xx, xx), xx);
        const Fp t = quad_mul(role == 0 ? p : role == 1 ? twice : role == 2 ? p : m, role == 3 ? m : v);
        // layer 3: M (S - X3) | W Y | - | W ZZZ, with X3 = M^2 - 2 S
        const Fp sx = shfl_fp(t, quad), mm = shfl_fp(t, quad + 3), w = shfl_fp(t, quad + 1);
        const Fp x3 = sub(mm, add(sx, sx));
        const Fp f = quad_mul(role == 0 ? m : p, role == 0 ? sub(sx, x3) : w);
        const Fp first = shfl_fp(f, quad);
        return role == 0 ? x3 : role == 1 ? sub(first, f) : role == 2 ? t : f;
    }

    // x (lane 0) and y (lane 1) of the affine point, Montgomery; (0, 0) for the point at infinity.  All quads of the
    // warp must hold points; called by whole warps.
    __device__ __forceinline__ Fp quad_to_affine(const Fp& p)
    {
        const int lane = threadIdx.x & 31, quad = lane & ~3, role = lane & 3;
        const Fp zz = shfl_fp(p, quad + 2), zzz = shfl_fp(p, quad + 3);
        const Fp inverse = inv_quad<FpCfg>(quad_mul(zz, zzz));  // 0 for the point at infinity
        return quad_mul(p, quad_mul(inverse, select_fp(role == 0, zzz, zz)));
    }
#endif
}
