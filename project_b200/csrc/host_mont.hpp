// Montgomery arithmetic on 64-bit limbs for the host side of the library.  A 32-bit carry flag has to be
// emulated there (a multiplication on it takes 2 us); the 64 x 64 -> 128 bit multiplier of the host does the
// same product in 30 to 80 ns.  Values lie in memory as the kernels' 32-bit limbs do (little-endian).
#pragma once

#include <cstdint>
#include <cstring>

namespace gzk
{
    template <typename Cfg>
    struct HostMont
    {
        static constexpr int W = Cfg::N / 2;
        using u128 = unsigned __int128;

        static constexpr uint64_t modulus(int i) { return static_cast<uint64_t>(Cfg::mod(2 * i + 1)) << 32 | Cfg::mod(2 * i); }
        // -modulus^-1 mod 2^64 from the 32-bit constant by one Newton step
        static constexpr uint64_t neg_inverse()
        {
            const uint64_t inv32 = 0u - Cfg::INV;
            return 0u - inv32 * (2u - modulus(0) * inv32);
        }

        // out = a - modulus where a + top 2^(64 W) >= modulus, else a
        static void reduce_once(const uint64_t* a, uint64_t top, uint64_t* out)
        {
            uint64_t d[W], borrow = 0;
            for (int i = 0; i < W; ++i)
            {
                const u128 t = static_cast<u128>(a[i]) - modulus(i) - borrow;
                d[i] = static_cast<uint64_t>(t);
                borrow = static_cast<uint64_t>(t >> 64) & 1u;
            }
            const bool keep = top == 0 && borrow != 0;
            for (int i = 0; i < W; ++i) out[i] = keep ? a[i] : d[i];
        }

        // Both carry chains of a row run side by side; `top` takes what two carries may exceed one limb by.
        static void mul(const void* pa, const void* pb, void* po)
        {
            uint64_t a[W], b[W], t[W] = {}, top = 0;
            std::memcpy(a, pa, sizeof(a));
            std::memcpy(b, pb, sizeof(b));
            for (int i = 0; i < W; ++i)
            {
                u128 x = static_cast<u128>(a[0]) * b[i] + t[0];
                const uint64_t m = static_cast<uint64_t>(x) * neg_inverse();
                u128 y = static_cast<u128>(m) * modulus(0) + static_cast<uint64_t>(x);
                for (int j = 1; j < W; ++j)
                {
                    x = static_cast<u128>(a[j]) * b[i] + t[j] + static_cast<uint64_t>(x >> 64);
                    y = static_cast<u128>(m) * modulus(j) + static_cast<uint64_t>(x) + static_cast<uint64_t>(y >> 64);
                    t[j - 1] = static_cast<uint64_t>(y);
                }
                const u128 last = static_cast<u128>(top) + static_cast<uint64_t>(x >> 64) + static_cast<uint64_t>(y >> 64);
                t[W - 1] = static_cast<uint64_t>(last);
                top = static_cast<uint64_t>(last >> 64);
            }
            uint64_t o[W];
            reduce_once(t, top, o);
            std::memcpy(po, o, sizeof(o));
        }

        static void add(const void* pa, const void* pb, void* po)
        {
            uint64_t a[W], b[W], s[W], o[W];
            std::memcpy(a, pa, sizeof(a));
            std::memcpy(b, pb, sizeof(b));
            u128 c = 0;
            for (int i = 0; i < W; ++i)
            {
                c += static_cast<u128>(a[i]) + b[i];
                s[i] = static_cast<uint64_t>(c);
                c >>= 64;
            }
            reduce_once(s, static_cast<uint64_t>(c), o);
            std::memcpy(po, o, sizeof(o));
        }

        static void sub(const void* pa, const void* pb, void* po)
        {
            uint64_t a[W], b[W], d[W], borrow = 0;
            std::memcpy(a, pa, sizeof(a));
            std::memcpy(b, pb, sizeof(b));
            for (int i = 0; i < W; ++i)
            {
                const u128 t = static_cast<u128>(a[i]) - b[i] - borrow;
                d[i] = static_cast<uint64_t>(t);
                borrow = static_cast<uint64_t>(t >> 64) & 1u;
            }
            const uint64_t mask = 0u - borrow;
            u128 c = 0;
            for (int i = 0; i < W; ++i)
            {
                c += static_cast<u128>(d[i]) + (modulus(i) & mask);
                d[i] = static_cast<uint64_t>(c);
                c >>= 64;
            }
            std::memcpy(po, d, sizeof(d));
        }
    };
}
