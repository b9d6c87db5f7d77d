// Field inversion as four cooperating lanes: every batch inversion, every commitment's affine
// conversion ends in one inversion that the rest of its CTA waits for, so what counts is its
// length as a dependent chain.
//
// Division steps in the "half-delta" form (Bernstein and Yang, "Fast constant-time gcd
// computation and modular inversion", 2019; the variant with delta starting at 1/2 needs at most
// (45907 bits + 26313) / 19929 steps): 30 of them run on the low words of f and g alone and are
// recorded as a 2 x 2 matrix of factors with |row| <= 2^30, which is then applied to the full-length
// f, g and to their cofactors d, e (f = d x, g = e x modulo the modulus).  Nothing is compared, so
// unlike the binary GCD with approximations a step needs neither the top words nor 64-bit
// arithmetic.  The four length-N updates of a round are independent
// and have the same shape, so each lane of a quad makes one of them:
//
//   role 0: f' = (u f + v g) / 2^30        role 2: d' = (u d + v e) / 2^30 mod modulus
//   role 1: g' = (q f + r g) / 2^30        role 3: e' = (q d + r e) / 2^30 mod modulus
//
// 30 steps take 1150 cycles (1510 one at a time), the update of twelve limbs 350; a base-field inversion
// 44 k cycles, 23 us, where the one-thread binary GCD took 60 us.
//
// A lane holds its own value X and its partner's Y (exchanged with the neighbouring lane after
// each round).  Values are two's complement on N + 1 limbs; |f|, |g|, |d|, |e| stay <= modulus.
#pragma once

#include "field.cuh"

namespace gzk
{
    struct DivstepMatrix
    {
        int32_t u, v, q, r;
    };

    constexpr int kDivsteps = 30;

    template <typename Cfg>
    struct DivstepRounds
    {
        static constexpr int value = ((45907 * Cfg::BITS + 26313) / 19929 + kDivsteps) / kDivsteps;
    };

    // 30 division steps on the low words; *zeta = -(delta + 1/2) travels between the rounds (-1 at first).
    // The trailing zeros of g are so many steps at once.  With g odd the next zeta + 1 steps add f to g or not and never
    // exchange them, so up to three of them are one multiple w of f, w = -g / f mod 8 = -g f mod 8 (an odd f is its own
    // inverse there).  Eleven passes of the loop on average instead of thirty single steps: what a lone warp is
    // short of is instructions in sequence.  All lanes of a warp invert the same value, so the branches are uniform.
    GZK_HD DivstepMatrix divsteps_30(uint32_t f, uint32_t g, int32_t* zeta_io)
    {
        uint32_t u = 1, v = 0, q = 0, r = 1;
        int32_t zeta = *zeta_io, left = kDivsteps;
        for (;;)
        {
            const uint32_t sentinel = g | (0xffffffffu << left);
#if defined(__CUDA_ARCH__)
            const int zeros = __clz(static_cast<int>(__brev(sentinel)));
#else
            const int zeros = __builtin_ctz(sentinel);
#endif
            g >>= zeros;
            u <<= zeros;
            v <<= zeros;
            zeta -= zeros;
            left -= zeros;
            if (left == 0) break;
            if (zeta < 0)
            {
                const uint32_t tf = f, tu = u, tv = v;
                f = g;
                u = q;
                v = r;
                g = 0u - tf;
                q = 0u - tu;
                r = 0u - tv;
                zeta = -1 - zeta;
            }
            const int steps = zeta + 1 < left ? zeta + 1 : left;
            const uint32_t w = (0u - g * f) & (steps >= 3 ? 7u : (1u << steps) - 1u);
            g += f * w;
            q += u * w;
            r += v * w;
        }
        *zeta_io = zeta;
        DivstepMatrix m;
        m.u = static_cast<int32_t>(u);
        m.v = static_cast<int32_t>(v);
        m.q = static_cast<int32_t>(q);
        m.r = static_cast<int32_t>(r);
        return m;
    }

    // X = (cx X + cy Y) / 2^30, exactly (modular = false: the low 30 bits are zero) or modulo the modulus.
    // |cx| + |cy| <= 2^30, |X|, |Y| <= modulus, all two's complement on W = N + 1 limbs; |result| <= modulus.
    template <typename Cfg>
    GZK_HD void divstep_update(uint32_t* X, const uint32_t* Y, int32_t cx, int32_t cy, bool modular)
    {
        constexpr int N = Cfg::N, W = N + 1;
        static_assert(N % 2 == 0, "limb count must be even");
        // c X = |c| (X ^ m) + (|c| & m) with m the sign of c
        const uint32_t mx = static_cast<uint32_t>(cx >> 31), my = static_cast<uint32_t>(cy >> 31);
        const uint32_t ax = (static_cast<uint32_t>(cx) ^ mx) - mx, ay = (static_cast<uint32_t>(cy) ^ my) - my;
        uint32_t E[W], O[W];  // products on even and on odd limb boundaries
        O[0] = (ax & mx) + (ay & my);
#pragma unroll
        for (int j = 0; j < W; ++j)
        {
            const uint32_t x = X[j] ^ mx;
            uint32_t* acc = (j & 1) ? O : E;
            acc[j] = mp::mul_lo(x, ax);
            if (j + 1 < W) acc[j + 1] = mp::mul_hi(x, ax);
        }
        E[0] = mp::mad_lo_cc(Y[0] ^ my, ay, E[0]);
        E[1] = mp::madc_hi_cc(Y[0] ^ my, ay, E[1]);
#pragma unroll
        for (int j = 2; j < W; j += 2)
        {
            E[j] = mp::madc_lo_cc(Y[j] ^ my, ay, E[j]);
            if (j + 1 < W) E[j + 1] = mp::madc_hi_cc(Y[j] ^ my, ay, E[j + 1]);
        }
        O[1] = mp::mad_lo_cc(Y[1] ^ my, ay, O[1]);
        O[2] = mp::madc_hi_cc(Y[1] ^ my, ay, O[2]);
#pragma unroll
        for (int j = 3; j < W; j += 2)
        {
            O[j] = mp::madc_lo_cc(Y[j] ^ my, ay, O[j]);
            O[j + 1] = mp::madc_hi_cc(Y[j] ^ my, ay, O[j + 1]);
        }
        E[0] = mp::add_cc(E[0], O[0]);
#pragma unroll
        for (int j = 1; j < W - 1; ++j) E[j] = mp::addc_cc(E[j], O[j]);
        E[W - 1] = mp::addc(E[W - 1], O[W - 1]);
        // the multiple of the modulus that clears the low 30 bits, of the sign that keeps |result| <= modulus
        {
            constexpr uint32_t M30 = (1u << kDivsteps) - 1u;
            const uint32_t k = (E[0] * Cfg::INV) & M30;
            const bool negative = (E[W - 1] >> 31) != 0;
            const uint32_t ak = modular ? (negative ? k : (1u << kDivsteps) - k) : 0u;
            const uint32_t mk = modular && !negative ? 0xffffffffu : 0u;
            uint32_t P[W];
#pragma unroll
            for (int j = 0; j < N; ++j) P[j] = Cfg::mod(j) ^ mk;
            P[W - 1] = mk;
            E[0] = mp::mad_lo_cc(P[0], ak, E[0]);
            E[1] = mp::madc_hi_cc(P[0], ak, E[1]);
#pragma unroll
            for (int j = 2; j < W; j += 2)
            {
                E[j] = mp::madc_lo_cc(P[j], ak, E[j]);
                if (j + 1 < W) E[j + 1] = mp::madc_hi_cc(P[j], ak, E[j + 1]);
            }
            O[0] = ak & mk;
            O[1] = mp::mul_lo(P[1], ak);
            O[2] = mp::mul_hi(P[1], ak);
#pragma unroll
            for (int j = 3; j < W; j += 2)
            {
                O[j] = mp::mul_lo(P[j], ak);
                O[j + 1] = mp::mul_hi(P[j], ak);
            }
            E[0] = mp::add_cc(E[0], O[0]);
#pragma unroll
            for (int j = 1; j < W - 1; ++j) E[j] = mp::addc_cc(E[j], O[j]);
            E[W - 1] = mp::addc(E[W - 1], O[W - 1]);
        }
#pragma unroll
        for (int j = 0; j < N; ++j) X[j] = (E[j] >> kDivsteps) | (E[j + 1] << (32 - kDivsteps));
        X[N] = static_cast<uint32_t>(static_cast<int32_t>(E[N]) >> kDivsteps);
    }

    // Start values of a role.  The cofactors start from R^2, so that for x = A R the result is A^-1 R.
    template <typename Cfg>
    GZK_HD void divstep_start(const Fe<Cfg>& value, int role, uint32_t* X, uint32_t* Y)
    {
        constexpr int N = Cfg::N;
#pragma unroll
        for (int i = 0; i < N; ++i)
        {
            const uint32_t first = role < 2 ? Cfg::mod(i) : 0u, second = role < 2 ? value.l[i] : Cfg::r2(i);
            X[i] = (role & 1) ? second : first;
            Y[i] = (role & 1) ? first : second;
        }
        X[N] = 0;
        Y[N] = 0;
    }

    // The inverse from the last d (two's complement, |d| <= modulus) and the sign of the last f (= +-1).
    template <typename Cfg>
    GZK_HD Fe<Cfg> divstep_result(const uint32_t* d, bool f_negative)
    {
        constexpr int N = Cfg::N;
        const uint32_t m = f_negative ? 0xffffffffu : 0u;
        Fe<Cfg> o;
        o.l[0] = mp::add_cc(d[0] ^ m, f_negative ? 1u : 0u);
#pragma unroll
        for (int i = 1; i < N; ++i) o.l[i] = mp::addc_cc(d[i] ^ m, 0);
        const uint32_t top = mp::addc(d[N] ^ m, 0);
        const uint32_t low = static_cast<uint32_t>(static_cast<int32_t>(top) >> 31);
        o.l[0] = mp::add_cc(o.l[0], low & Cfg::mod(0));
#pragma unroll
        for (int i = 1; i < N - 1; ++i) o.l[i] = mp::addc_cc(o.l[i], low & Cfg::mod(i));
        o.l[N - 1] = mp::addc(o.l[N - 1], low & Cfg::mod(N - 1));
        return reduce_once(o);
    }

    // The four roles one after another (the arithmetic of inv_quad() for checks on the host).
    template <typename Cfg>
    GZK_HD Fe<Cfg> inv_divsteps(const Fe<Cfg>& value)
    {
        constexpr int N = Cfg::N;
        uint32_t X[4][N + 1], Y[4][N + 1];
        for (int role = 0; role < 4; ++role) divstep_start<Cfg>(value, role, X[role], Y[role]);
        int32_t zeta = -1;
        for (int round = 0; round < DivstepRounds<Cfg>::value; ++round)
        {
            const DivstepMatrix m = divsteps_30(X[0][0], X[1][0], &zeta);
            for (int role = 0; role < 4; ++role)
                divstep_update<Cfg>(X[role], Y[role], (role & 1) ? m.r : m.u, (role & 1) ? m.q : m.v, role >= 2);
            uint32_t any = 0;
            for (int i = 0; i <= N; ++i)
            {
                for (int role = 0; role < 4; ++role) Y[role][i] = X[role ^ 1][i];
                any |= X[1][i];
            }
            if (any == 0) break;
        }
        return divstep_result<Cfg>(X[2], (X[0][N] >> 31) != 0);
    }

#if defined(__CUDACC__)
    // Inverse of `value` (Montgomery in and out, 0 for 0): called by whole warps whose lanes all pass the same value.
    template <typename Cfg>
    __device__ __noinline__ Fe<Cfg> inv_quad(const Fe<Cfg> value)
    {
        constexpr int N = Cfg::N;
        const int lane = threadIdx.x & 31, role = lane & 3, quad = lane & ~3;
        uint32_t X[N + 1], Y[N + 1];
        divstep_start<Cfg>(value, role, X, Y);
        int32_t zeta = -1;
#pragma unroll 1
        for (int round = 0; round < DivstepRounds<Cfg>::value; ++round)
        {
            const uint32_t f0 = __shfl_sync(0xffffffffu, X[0], quad), g0 = __shfl_sync(0xffffffffu, X[0], quad + 1);
            const DivstepMatrix m = divsteps_30(f0, g0, &zeta);
            divstep_update<Cfg>(X, Y, (role & 1) ? m.r : m.u, (role & 1) ? m.q : m.v, role >= 2);
            uint32_t any = 0;
#pragma unroll
            for (int i = 0; i <= N; ++i)
            {
                Y[i] = __shfl_xor_sync(0xffffffffu, X[i], 1);
                any |= X[i];
            }
            if (!__any_sync(0xffffffffu, role == 1 && any != 0)) break;
        }
        const bool f_negative = (__shfl_sync(0xffffffffu, X[N], quad) >> 31) != 0;
#pragma unroll
        for (int i = 0; i <= N; ++i) X[i] = __shfl_sync(0xffffffffu, X[i], quad + 2);
        return divstep_result<Cfg>(X, f_negative);
    }
#endif
}
