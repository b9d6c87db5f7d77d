// Host-side check of the division-step inversion (the four lane roles run one after another)
// against the oracle: random values, small ones, single bits and the modulus minus them.
#include <cstdio>
#include <cstring>
#include <random>

#include "../../oracle/field.hpp"
#include "../../project_b200/csrc/inverse.cuh"

template <typename Cfg, typename OFe, size_t N64>
int check(const char* name, std::mt19937_64& rng)
{
    int failures = 0;
    auto one = [&](const oracle::BigInt<N64>& c) {
        if (oracle::cmp(c, OFe::P().modulus) >= 0) return;
        OFe o;
        o.v = c;  // taken as a Montgomery representation: any residue is one
        gzk::Fe<Cfg> f;
        std::memcpy(f.l, c.w.data(), 4 * Cfg::N);
        const gzk::Fe<Cfg> got = gzk::inv_divsteps(f);
        const OFe want = o.is_zero() ? o : o.inv();
        if (std::memcmp(got.l, want.v.w.data(), 4 * Cfg::N) != 0 && ++failures < 5) std::printf("%s inverse mismatch\n", name);
    };
    auto minus = [&](const oracle::BigInt<N64>& c) {
        oracle::BigInt<N64> d{};
        unsigned __int128 borrow = 0;
        for (size_t i = 0; i < N64; ++i)
        {
            const unsigned __int128 w = static_cast<unsigned __int128>(OFe::P().modulus.w[i]) - c.w[i] - borrow;
            d.w[i] = static_cast<uint64_t>(w);
            borrow = (w >> 64) & 1;
        }
        return d;
    };
    for (int iter = 0; iter < 20000; ++iter)
    {
        oracle::BigInt<N64> c;
        for (auto& w : c.w) w = rng();
        c.w[N64 - 1] &= (~0ULL) >> (64 * N64 - OFe::P().modulus.bit_length());
        one(c);
    }
    for (uint64_t small = 0; small < 300; ++small)
    {
        oracle::BigInt<N64> c{};
        c.w[0] = small;
        one(c);
        if (small != 0) one(minus(c));
    }
    for (int bit = 0; bit < Cfg::BITS; ++bit)
    {
        oracle::BigInt<N64> c{}, ones{};
        c.w[bit / 64] = 1ULL << (bit % 64);
        one(c);
        one(minus(c));
        for (int b = 0; b <= bit; ++b) ones.w[b / 64] |= 1ULL << (b % 64);
        one(ones);
    }
    return failures;
}

int main()
{
    std::mt19937_64 rng(4242);
    const int failures = check<gzk::FrCfg, oracle::Fr, 4>("Fr", rng) + check<gzk::FpCfg, oracle::Fp, 6>("Fp", rng);
    std::printf(failures == 0 ? "OK\n" : "FAILED %d\n", failures);
    return failures == 0 ? 0 : 1;
}
