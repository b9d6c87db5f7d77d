// The 64-bit host point arithmetic against the formulas of the kernels (themselves checked against the oracle):
// sums, doublings, opposite and coinciding operands, infinities, the Horner sum over windows.
#include <cstdio>
#include <cstring>
#include <random>

#include "../../project_b200/csrc/host_g1.hpp"

static gzk::HostXyzz to_host(const gzk::G1Xyzz& p)
{
    gzk::HostXyzz h;
    std::memcpy(&h, &p, sizeof(h));
    return h;
}
static bool same(const gzk::HostXyzz& h, const gzk::G1Xyzz& p)
{
    uint8_t a[96], b[96] = {};
    gzk::host_to_affine_bytes(h, a);
    const gzk::G1Affine q = gzk::g1_to_affine(p);
    const gzk::Fp x = gzk::from_mont(q.x), y = gzk::from_mont(q.y);
    std::memcpy(b, x.l, 48);
    std::memcpy(b + 48, y.l, 48);
    return std::memcmp(a, b, 96) == 0;
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
    for (int i = 0; i < 24; ++i)
    {
        if (!same(gzk::host_double(to_host(pool[i])), gzk::g1_double(pool[i]))) ++failures;
        for (int j = 0; j < 24; ++j)
            if (!same(gzk::host_add(to_host(pool[i]), to_host(pool[j])), gzk::g1_add(pool[i], pool[j]))) ++failures;
    }
    for (unsigned c : {1u, 7u, 16u})
        for (size_t count : {1u, 2u, 24u})
        {
            gzk::HostXyzz points[24];
            gzk::G1Xyzz want = gzk::G1Xyzz::infinity();
            for (size_t w = count; w-- > 0;)
            {
                points[w] = to_host(pool[w]);
                for (unsigned k = 0; k < c; ++k) want = gzk::g1_double(want);
                want = gzk::g1_add(want, pool[w]);
            }
            if (!same(gzk::host_horner(points, count, c), want)) ++failures;
        }
    for (int i = 0; i < 20000; ++i)
    {
        gzk::HostFp a, b;
        for (int k = 0; k < 6; ++k)
        {
            a.w[k] = i % 5 == 0 ? gzk::host_fp::modulus(k) : rng();
            b.w[k] = i % 7 == 0 ? gzk::host_fp::modulus(k) : rng();
        }
        a.w[5] = i % 5 == 0 ? a.w[5] : a.w[5] % gzk::host_fp::modulus(5);
        b.w[5] = i % 7 == 0 ? b.w[5] : b.w[5] % gzk::host_fp::modulus(5);
        if (i % 5 == 0) a.w[0] -= 1 + rng() % 3;
        if (i % 7 == 0) b.w[0] -= 1 + rng() % 3;
        gzk::Fp fa, fb;
        std::memcpy(fa.l, a.w, 48);
        std::memcpy(fb.l, b.w, 48);
        const gzk::HostFp p = gzk::host_fp::mul(a, b), s = gzk::host_fp::add(a, b), d = gzk::host_fp::sub(a, b);
        if (std::memcmp(p.w, gzk::mul(fa, fb).l, 48) != 0 || std::memcmp(s.w, gzk::add(fa, fb).l, 48) != 0 || std::memcmp(d.w, gzk::sub(fa, fb).l, 48) != 0) ++failures;
    }
    std::printf(failures == 0 ? "OK\n" : "FAILED %d\n", failures);
    return failures == 0 ? 0 : 1;
}
