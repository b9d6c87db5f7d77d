// Base-field and point arithmetic for the host on six 64-bit limbs (the memory layout of the twelve
// 32-bit limbs of the kernels, Montgomery form with R = 2^384).  For chains that are serial whatever
// they run on: a multiplication takes about 40 ns here and 600 ns as the only work of a warp.
#pragma once

#include <cstdint>
#include <cstring>

#include "g1.cuh"

namespace gzk
{
    struct HostFp
    {
        uint64_t w[6];
    };

    namespace host_fp
    {
        constexpr uint64_t modulus(int i) { return static_cast<uint64_t>(FpCfg::mod(2 * i + 1)) << 32 | FpCfg::mod(2 * i); }

        // -p^-1 mod 2^64 from the 32-bit constant by one Newton step
        constexpr uint64_t neg_inverse()
        {
            const uint64_t inv32 = 0u - FpCfg::INV;  // p^-1 mod 2^32
            return 0u - inv32 * (2u - modulus(0) * inv32);
        }

        inline bool is_zero(const HostFp& a) { return (a.w[0] | a.w[1] | a.w[2] | a.w[3] | a.w[4] | a.w[5]) == 0; }

        // a - p where a >= p (a < 2p)
        inline HostFp reduce_once(const HostFp& a)
        {
            HostFp d;
            unsigned __int128 borrow = 0;
            for (int i = 0; i < 6; ++i)
            {
                const unsigned __int128 t = static_cast<unsigned __int128>(a.w[i]) - modulus(i) - borrow;
                d.w[i] = static_cast<uint64_t>(t);
                borrow = (t >> 64) & 1;
            }
            return borrow ? a : d;
        }

        inline HostFp add(const HostFp& a, const HostFp& b)
        {
            HostFp s;
            unsigned __int128 carry = 0;
            for (int i = 0; i < 6; ++i)
            {
                carry += static_cast<unsigned __int128>(a.w[i]) + b.w[i];
                s.w[i] = static_cast<uint64_t>(carry);
                carry >>= 64;
            }
            return reduce_once(s);
        }

        inline HostFp sub(const HostFp& a, const HostFp& b)
        {
            HostFp d;
            unsigned __int128 borrow = 0;
            for (int i = 0; i < 6; ++i)
            {
                const unsigned __int128 t = static_cast<unsigned __int128>(a.w[i]) - b.w[i] - borrow;
                d.w[i] = static_cast<uint64_t>(t);
                borrow = (t >> 64) & 1;
            }
            const uint64_t mask = borrow ? ~0ull : 0ull;
            unsigned __int128 carry = 0;
            for (int i = 0; i < 6; ++i)
            {
                carry += static_cast<unsigned __int128>(d.w[i]) + (modulus(i) & mask);
                d.w[i] = static_cast<uint64_t>(carry);
                carry >>= 64;
            }
            return d;
        }

        // Montgomery product; both carry chains of a row run side by side.  The top limb of p is below 2^62, so
        // the sum of the two carries fits one limb.
        inline HostFp mul(const HostFp& a, const HostFp& b)
        {
            using u128 = unsigned __int128;
            const uint64_t inv = neg_inverse();
            uint64_t t[6] = {};
            for (int i = 0; i < 6; ++i)
            {
                u128 x = static_cast<u128>(a.w[0]) * b.w[i] + t[0];
                const uint64_t m = static_cast<uint64_t>(x) * inv;
                u128 y = static_cast<u128>(m) * modulus(0) + static_cast<uint64_t>(x);
                for (int j = 1; j < 6; ++j)
                {
                    x = static_cast<u128>(a.w[j]) * b.w[i] + t[j] + static_cast<uint64_t>(x >> 64);
                    y = static_cast<u128>(m) * modulus(j) + static_cast<uint64_t>(x) + static_cast<uint64_t>(y >> 64);
                    t[j - 1] = static_cast<uint64_t>(y);
                }
                t[5] = static_cast<uint64_t>(x >> 64) + static_cast<uint64_t>(y >> 64);
            }
            HostFp r;
            std::memcpy(r.w, t, sizeof(r.w));
            return reduce_once(r);
        }
    }

    struct HostXyzz
    {
        HostFp X, Y, ZZ, ZZZ;
        bool is_infinity() const { return host_fp::is_zero(ZZ); }
    };
    static_assert(sizeof(HostXyzz) == sizeof(G1Xyzz), "device points are read as they lie in memory");

    inline HostXyzz host_double(const HostXyzz& p)
    {
        using namespace host_fp;
        if (p.is_infinity()) return p;
        const HostFp U = add(p.Y, p.Y), V = mul(U, U), W = mul(U, V), S = mul(p.X, V), xx = mul(p.X, p.X), M = add(add(xx, xx), xx);
        HostXyzz r;
        r.X = sub(mul(M, M), add(S, S));
        r.Y = sub(mul(M, sub(S, r.X)), mul(W, p.Y));
        r.ZZ = mul(V, p.ZZ);
        r.ZZZ = mul(W, p.ZZZ);
        return r;
    }

    inline HostXyzz host_add(const HostXyzz& p, const HostXyzz& q)
    {
        using namespace host_fp;
        if (p.is_infinity()) return q;
        if (q.is_infinity()) return p;
        const HostFp U1 = mul(p.X, q.ZZ), S1 = mul(p.Y, q.ZZZ);
        const HostFp P = sub(mul(q.X, p.ZZ), U1), R = sub(mul(q.Y, p.ZZZ), S1);
        if (host_fp::is_zero(P))
        {
            if (host_fp::is_zero(R)) return host_double(p);
            return HostXyzz{};
        }
        const HostFp PP = mul(P, P), PPP = mul(P, PP), Q = mul(U1, PP);
        HostXyzz r;
        r.X = sub(sub(mul(R, R), PPP), add(Q, Q));
        r.Y = sub(mul(R, sub(Q, r.X)), mul(S1, PPP));
        r.ZZ = mul(mul(p.ZZ, q.ZZ), PP);
        r.ZZZ = mul(mul(p.ZZZ, q.ZZZ), PPP);
        return r;
    }

    // Canonical affine coordinates in wire format (96 zero bytes for the point at infinity)
    inline void host_to_affine_bytes(const HostXyzz& p, uint8_t out[96])
    {
        using namespace host_fp;
        std::memset(out, 0, 96);
        if (p.is_infinity()) return;
        const HostFp z = mul(p.ZZ, p.ZZZ);
        Fp zd;
        std::memcpy(zd.l, z.w, 48);
        zd = inv(zd);
        HostFp zi;
        std::memcpy(zi.w, zd.l, 48);
        const HostFp one{{1, 0, 0, 0, 0, 0}};
        const HostFp x = mul(mul(p.X, mul(zi, p.ZZZ)), one), y = mul(mul(p.Y, mul(zi, p.ZZ)), one);
        std::memcpy(out, x.w, 48);
        std::memcpy(out + 48, y.w, 48);
    }

    // sum_w 2^(c w) points[w], `count` > 0 of them
    inline HostXyzz host_horner(const HostXyzz* points, size_t count, unsigned c)
    {
        HostXyzz acc = points[count - 1];
        for (size_t w = count - 1; w-- > 0;)
        {
            for (unsigned k = 0; k < c; ++k) acc = host_double(acc);
            acc = host_add(acc, points[w]);
        }
        return acc;
    }
}
