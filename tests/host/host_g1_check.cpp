// The 64-bit host arithmetic against the carry chains of the kernels (themselves checked against the oracle), and the
// Horner sum over windows.
#include <cstdio>
#include <cstring>
#include <random>

#include "../../project_b200/csrc/host_g1.hpp"

static bool same(const gzk::G1Xyzz& h, const gzk::G1Xyzz& p)
{
    uint8_t a[96], b[96] = {};
    gzk::host_to_affine_bytes(h, a);
    const gzk::G1Affine q = gzk::g1_to_affine(p);
    const gzk::Fp x = gzk::from_mont(q.x), y = gzk::from_mont(q.y);
    std::memcpy(b, x.l, 48);
    std::memcpy(b + 48, y.l, 48);
    return std::memcmp(a, b, 96) == 0;
}

// 64-bit products, sums and differences against the carry chains, with the extremes of the field among the values
template <typename Cfg>
int check_limbs(std::mt19937_64& rng)
{
    using F = gzk::Fe<Cfg>;
    int failures = 0;
    auto value = [&]() {
        F f = F::modulus();
        switch (rng() % 8)
        {
        case 0: f.l[0] -= 1 + static_cast<uint32_t>(rng() % 4 == 0 ? 0 : f.l[0] > 4 ? rng() % 3 : 0); return f;
        case 1: f = F::zero(); f.l[0] = static_cast<uint32_t>(rng() % 3); return f;
        default:
            for (int i = 0; i < Cfg::N; ++i) f.l[i] = static_cast<uint32_t>(rng());
            f.l[Cfg::N - 1] %= Cfg::mod(Cfg::N - 1);
            return f;
        }
    };
    for (int i = 0; i < 40000; ++i)
    {
        const F a = value(), b = value();
        F m, s, d;
        gzk::HostMont<Cfg>::mul(a.l, b.l, m.l);
        gzk::HostMont<Cfg>::add(a.l, b.l, s.l);
        gzk::HostMont<Cfg>::sub(a.l, b.l, d.l);
        if (m != gzk::mul(a, b) || s != gzk::add(a, b) || d != gzk::sub(a, b)) ++failures;
    }
    return failures;
}

int main()
{
    std::mt19937_64 rng(99);
    int failures = 0;
    gzk::G1Affine g;  // the generator from its published coordinates
    auto parse = [](const char* hex) {
        gzk::Fp f;
        for (int i = 0; i < 12; ++i) std::sscanf(hex + 8 * (11 - i), "%8x", &f.l[i]);
        return gzk::to_mont(f);
    };
    g.x = parse("17f1d3a73197d7942695638c4fa9ac0fc3688c4f9774b905a14e3a3f171bac586c55e83ff97a1aeffb3af00adb22c6bb");
    g.y = parse("08b3f481e3aaa0f1a09e30ed741d8ae4fcf5e095d5d00af600db18cb2c04b3edd03cc744a2888ae40caa232946c5e7e1");
    gzk::G1Xyzz pool[24];
    pool[0] = gzk::G1Xyzz::infinity();
    pool[1] = gzk::G1Xyzz::from_affine(g);
    pool[2] = pool[1];
    pool[2].Y = gzk::neg(pool[2].Y);
    for (int i = 3; i < 24; ++i) pool[i] = rng() % 2 ? gzk::g1_double(pool[rng() % i]) : gzk::g1_add(pool[rng() % i], pool[rng() % i]);
    for (unsigned c : {1u, 7u, 16u})
        for (size_t count : {1u, 2u, 24u})
        {
            gzk::G1Xyzz points[24];
            gzk::G1Xyzz want = gzk::G1Xyzz::infinity();
            for (size_t w = count; w-- > 0;)
            {
                points[w] = pool[w];
                for (unsigned k = 0; k < c; ++k) want = gzk::g1_double(want);
                want = gzk::g1_add(want, pool[w]);
            }
            if (!same(gzk::host_horner(points, count, c), want)) ++failures;
        }
    failures += check_limbs<gzk::FrCfg>(rng) + check_limbs<gzk::FpCfg>(rng);
    std::printf(failures == 0 ? "OK\n" : "FAILED %d\n", failures);
    return failures == 0 ? 0 : 1;
}
