// Stand-alone Fr NTT / inverse NTT / coset variants and the multilinear fold
// (kernel sweep; the reference has no transform on its proving path).
//
// Natural order in, natural order out.  The log2(n) radix-2 stages are grouped into
// passes (10 stages in the first, up to 8 in the others); each pass holds a
// 1024-element tile, four elements per thread, in registers, runs two stages on them and passes the
// tile through shared memory (limb-planar, conflict-free) to the next two, and writes it back, so a
// 2^24-point transform touches HBM in 3 passes instead of 24.  Pass 0 gathers its tile through the
// bit-reversal permutation; later passes take tiles of 2^S strided rows by 2^(10-S) contiguous
// elements (S <= 8, at least one 128-byte line per row).  Calls that would leave SMs without a
// tile take tiles of 256 elements (8 stages, then up to 6) on CTAs of 64 threads.
//
// Twiddles.  The stage-s butterfly of element pair (.., j) needs omega_(2^(s+1))^j with
// j the low s bits of the index.  Inside a pass that starts at stage s0, j splits into the
// bits below s0 ("low", constant through the pass) and the bits of the tile row that the
// pass has already combined, m: omega_(2^(s+1))^j = omega_(2^(t+1))^m * omega_(2^(s+1))^low
// with t = s - s0.  Multiplying element (row, low) ONCE, on load, by
// omega_(2^(s0+S))^(low * bitrev_S(row)) removes the second factor from every stage of the
// pass (the factor a row still carries after stage t is exactly what the remaining stages
// expect), so the stages use only the first factor: a 1024th root of unity from a
// 512-entry table, one multiplication per butterfly and none where m = 0.  The load-time
// factors come from a table per (s0, S) built once per context ([bitrev row][low], so a
// warp reads it in the same runs as the data); above 2^25 entries they are generated
// from the two-level omega tables instead (one more multiplication per element).
#include <cstdlib>
#include <cstring>

#include "block.cuh"

namespace gzk
{
    namespace
    {
        constexpr int kThreads = 256;
        constexpr int kTileBits = 10;
        constexpr int kSmallTileBits = 8;

        struct NttArgs
        {
            ColRef in;          // pass 0 only
            uint64_t in_count;  // elements stored per vector; the rest of its n are zeros
            Fr* data;           // output / in-place working vector (Montgomery)
            const Fr* small;    // omega_1024^m (or the inverse powers), m < 512: in-pass twiddles
            const Fr* twist;    // pass > 0: load-time factors [bitrev row][low]; NULL = generate them
            const Fr* lo;       // omega^j or omega^-j (generated load-time factors)
            const Fr* hi;
            unsigned lo_bits;
            unsigned log2n;
            unsigned s0;        // first stage of this pass
            unsigned stages;    // stages in this pass
            unsigned low_bits;  // contiguous low bits in the tile (L)
            int scale_mode;     // 0 none, 1 multiply the output by `scale` (1/n), 2 output i by the i-th entry of the shift tables
            Fr scale;
            const Fr* shift_lo; // powers of the coset shift (times 1/n where the output takes them)
            const Fr* shift_hi;
            unsigned shift_lo_bits;
            int pre_shift;      // pass 0: multiply input i by the i-th entry of the shift tables
        };

        // Word of element e in a limb plane.  In a round on bits pos, pos + 1 a warp's lanes run over five of the bits
        // 0 .. 6 of e that leave those two out; folding bits 5 and 6 onto alternating bank bits keeps the 32 lanes on
        // 32 banks for every pos.
        __device__ __forceinline__ uint32_t tile_word(uint32_t e) { return e ^ ((e >> 5) & 1u) * 0x0au ^ ((e >> 6) & 1u) * 0x15u; }
        template <int TILE>
        __device__ __forceinline__ void smem_store(uint32_t* tile, uint32_t e, const Fr& v)
        {
            const uint32_t w = tile_word(e);
#pragma unroll
            for (int i = 0; i < 8; ++i) tile[i * TILE + w] = v.l[i];
        }
        template <int TILE>
        __device__ __forceinline__ Fr smem_load(const uint32_t* tile, uint32_t e)
        {
            const uint32_t w = tile_word(e);
            Fr v;
#pragma unroll
            for (int i = 0; i < 8; ++i) v.l[i] = tile[i * TILE + w];
            return v;
        }
        __device__ __forceinline__ uint64_t bit_reverse(uint64_t x, unsigned bits)
        {
            return bits == 0 ? 0 : (__brevll(x) >> (64 - bits));
        }

        // global index of tile element e: [high | mid (stages bits) | lowbase | l (low_bits)]
        __device__ __forceinline__ uint64_t tile_index(const NttArgs& a, uint64_t tile_id, uint32_t e)
        {
            const uint32_t l = e & ((1u << a.low_bits) - 1u);
            const uint32_t mid = e >> a.low_bits;
            const unsigned lowbase_bits = a.s0 - a.low_bits;
            const uint64_t lowbase = tile_id & ((1ULL << lowbase_bits) - 1ULL);
            const uint64_t high = tile_id >> lowbase_bits;
            return (high << (a.s0 + a.stages)) | (static_cast<uint64_t>(mid) << a.s0) | (lowbase << a.low_bits) | l;
        }

        __device__ __forceinline__ Fr ntt_load(const NttArgs& a, uint64_t vec, uint64_t tile_id, uint32_t e)
        {
            const uint64_t gi = tile_index(a, tile_id, e);
            Fr v;
            if (a.s0 == 0)
            {
                const uint64_t src = bit_reverse(gi, a.log2n);
                if (src >= a.in_count) return Fr::zero();
                const ColRef in = a.in;
                v = col_load_mont(in, vec * a.in_count + src);
                if (a.pre_shift) v = mul(v, domain_point(a.shift_lo, a.shift_hi, a.shift_lo_bits, src));
            }
            else
            {
                v = load_fr_plain(a.data + (vec << a.log2n) + gi);
                const uint32_t c = __brev(e >> a.low_bits) >> (32 - a.stages);
                const uint64_t low = gi & ((1ULL << a.s0) - 1ULL);
                if (c != 0 && low != 0)
                {
                    const Fr w = a.twist != nullptr ? load_fr(a.twist + ((static_cast<uint64_t>(c) << a.s0) | low))
                                                    : domain_point(a.lo, a.hi, a.lo_bits, (low * c) << (a.log2n - a.s0 - a.stages));
                    v = mul(v, w);
                }
            }
            return v;
        }
        __device__ __forceinline__ void ntt_store(const NttArgs& a, uint64_t vec, uint64_t tile_id, uint32_t e, Fr v)
        {
            const uint64_t gi = tile_index(a, tile_id, e);
            if (a.scale_mode == 1) v = mul(v, a.scale);
            if (a.scale_mode == 2) v = mul(v, domain_point(a.shift_lo, a.shift_hi, a.shift_lo_bits, gi));
            store_fr(a.data + (vec << a.log2n) + gi, v);
        }
        __device__ __forceinline__ void butterfly(Fr& x, Fr& y)
        {
            const Fr u = x;
            x = add(u, y);
            y = sub(u, y);
        }

        // A thread holds the four tile elements that differ in bits pos and pos + 1 and runs the two stages on them
        // (the last round of an odd number of stages: one stage, on bit pos + 1).  Between rounds the tile passes
        // through shared memory: half the shared-memory traffic and half the barriers of a stage at a time.
        // A round writes the words that the same thread alone read before, so one barrier per round is enough.
        // 2^22 points, inverse from a coset: 1303 -> 1135 us.
        template <int TILE_BITS>
        __global__ void __launch_bounds__((1 << TILE_BITS) / 4, TILE_BITS == kTileBits ? 3 : 8) ntt_pass_kernel(NttArgs a)
        {
            constexpr int TILE = 1 << TILE_BITS;
            __shared__ uint32_t tile[8 * TILE];
            const uint64_t vec = blockIdx.y;
            // Pass 0 gathers through the bit-reversal permutation: element e of tile T comes from
            // rev10(e) * n/1024 + rev(T), one 32-byte element per 128-byte line.  The four tiles T, T + Q,
            // T + 2Q, T + 3Q (Q = tiles / 4) read the four elements of the SAME lines, so they are given
            // to four consecutive CTAs: they run side by side and three of the four line reads hit L2
            // instead of DRAM.
            uint64_t tile_id = blockIdx.x;
            if (a.s0 == 0 && gridDim.x >= 4) tile_id = static_cast<uint64_t>(blockIdx.x & 3u) * (gridDim.x >> 2) + (blockIdx.x >> 2);
            if (a.stages + a.low_bits < 2)  // n = 1 or 2
            {
                Fr x = ntt_load(a, vec, tile_id, 0), y = Fr::zero();
                if (a.stages == 1)
                {
                    y = ntt_load(a, vec, tile_id, 1);
                    butterfly(x, y);
                    ntt_store(a, vec, tile_id, 1, y);
                }
                ntt_store(a, vec, tile_id, 0, x);
                return;
            }
            const uint32_t b = threadIdx.x;
            uint32_t pos = a.low_bits - (a.stages == 1 ? 1 : 0);
            auto element = [&](uint32_t k) { return ((b >> pos) << (pos + 2)) | (k << pos) | (b & ((1u << pos) - 1u)); };
            Fr v[4];
#pragma unroll
            for (uint32_t k = 0; k < 4; ++k) v[k] = ntt_load(a, vec, tile_id, element(k));
            for (unsigned t = 0;;)
            {
                // m: the rows below the stage's bit that the pass has combined already
                if (t + 2 <= a.stages)
                {
                    const uint32_t m = (b & ((1u << pos) - 1u)) >> a.low_bits;
                    if (m != 0)
                    {
                        const Fr w = load_fr(a.small + (m << (9 - t)));
                        v[1] = mul(v[1], w);
                        v[3] = mul(v[3], w);
                    }
                    butterfly(v[0], v[1]);
                    butterfly(v[2], v[3]);
                    if (m != 0) v[2] = mul(v[2], load_fr(a.small + (m << (8 - t))));
                    v[3] = mul(v[3], load_fr(a.small + ((m | (1u << t)) << (8 - t))));
                    butterfly(v[0], v[2]);
                    butterfly(v[1], v[3]);
                    t += 2;
                }
                else
                {
#pragma unroll
                    for (uint32_t k = 0; k < 2; ++k)
                    {
                        const uint32_t m = (element(k) & ((2u << pos) - 1u)) >> a.low_bits;
                        if (m != 0) v[2 + k] = mul(v[2 + k], load_fr(a.small + (m << (9 - t))));
                        butterfly(v[k], v[2 + k]);
                    }
                    ++t;
                }
                if (t == a.stages) break;
#pragma unroll
                for (uint32_t k = 0; k < 4; ++k) smem_store<TILE>(tile, element(k), v[k]);
                __syncthreads();
                pos = a.low_bits + t - (t + 1 == a.stages ? 1 : 0);
#pragma unroll
                for (uint32_t k = 0; k < 4; ++k) v[k] = smem_load<TILE>(tile, element(k));
            }
#pragma unroll
            for (uint32_t k = 0; k < 4; ++k) ntt_store(a, vec, tile_id, element(k), v[k]);
        }

        // lo[j] = base^j and hi[j] = factor * base^(j << lo_bits), from the squarings of the base
        struct PowerTableArgs
        {
            Fr square[32];  // base^(2^k)
            Fr factor;
            uint32_t lo_bits, hi_bits;
            Fr* lo;
            Fr* hi;
        };
        __global__ void power_tables_kernel(PowerTableArgs a)
        {
            uint32_t j = blockIdx.x * blockDim.x + threadIdx.x;
            const uint32_t lo_count = 1u << a.lo_bits, hi_count = 1u << a.hi_bits;
            if (j >= lo_count + hi_count) return;
            const bool high = j >= lo_count;
            if (high) j -= lo_count;
            const uint32_t first = high ? a.lo_bits : 0;
            Fr v = high ? a.factor : Fr::one();
#pragma unroll 1
            for (uint32_t k = 0; (j >> k) != 0; ++k)
                if ((j >> k) & 1u) v = mul(v, a.square[first + k]);
            store_fr((high ? a.hi : a.lo) + j, v);
        }

        // out[(c << s0) | low] = omega_(2^(s0+S))^(low * c): the load-time factors of a pass
        __global__ void twist_table_kernel(const Fr* lo, const Fr* hi, unsigned lo_bits, unsigned s0, uint64_t count, Fr* out)
        {
            const uint64_t i = static_cast<uint64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
            if (i >= count) return;
            const uint64_t low = i & ((1ULL << s0) - 1ULL), c = i >> s0;
            store_fr(out + i, domain_point(lo, hi, lo_bits, low * c));
        }
        __global__ void small_table_kernel(const Fr* lo, const Fr* hi, unsigned lo_bits, Fr* out)
        {
            const uint32_t m = blockIdx.x * blockDim.x + threadIdx.x;
            if (m < 512) store_fr(out + m, domain_point(lo, hi, lo_bits, m));
        }

        constexpr unsigned kTwistTableMaxBits = 25;  // 1 GiB of load-time factors at most per table

        // The in-pass twiddle table (omega_1024^(+-m)) of the context, built on first use.
        int small_table(gzk_ctx* ctx, bool inverse, const Fr** out)
        {
            Fr*& slot = ctx->ntt_small[inverse ? 1 : 0];
            if (slot == nullptr)
            {
                const DomainTables* dom = nullptr;
                int rc = get_domain(ctx, 10, &dom);
                if (rc != GZK_OK) return rc;
                GZK_CUDA_TRY(ctx, cudaMalloc(reinterpret_cast<void**>(&slot), 512 * sizeof(Fr)));
                small_table_kernel<<<4, 128, 0, ctx->stream>>>(inverse ? dom->lo_inv : dom->lo, inverse ? dom->hi_inv : dom->hi, dom->lo_bits, slot);
                GZK_CUDA_TRY(ctx, cudaGetLastError());
            }
            *out = slot;
            return GZK_OK;
        }

        // The load-time factor table of a pass (s0, stages), built on first use; *out = NULL
        // when the table would exceed the size limit (the kernel then generates the factors).
        int twist_table(gzk_ctx* ctx, unsigned s0, unsigned stages, bool inverse, const Fr** out)
        {
            *out = nullptr;
            if (s0 + stages > kTwistTableMaxBits) return GZK_OK;
            for (const NttTwistTable& t : ctx->ntt_twists)
                if (t.s0 == s0 && t.stages == stages && t.inverse == inverse)
                {
                    *out = t.table;
                    return GZK_OK;
                }
            const DomainTables* dom = nullptr;
            int rc = get_domain(ctx, s0 + stages, &dom);
            if (rc != GZK_OK) return rc;
            const uint64_t count = 1ULL << (s0 + stages);
            NttTwistTable entry;
            entry.s0 = s0;
            entry.stages = stages;
            entry.inverse = inverse;
            const cudaError_t err = cudaMalloc(reinterpret_cast<void**>(&entry.table), count * sizeof(Fr));
            if (err != cudaSuccess)
            {
                cudaGetLastError();  // no room for the table: fall back to generated factors
                return GZK_OK;
            }
            twist_table_kernel<<<static_cast<unsigned>((count + 255) / 256), 256, 0, ctx->stream>>>(
                inverse ? dom->lo_inv : dom->lo, inverse ? dom->hi_inv : dom->hi, dom->lo_bits, s0, count, entry.table);
            GZK_CUDA_TRY(ctx, cudaGetLastError());
            ctx->ntt_twists.push_back(entry);
            *out = entry.table;
            return GZK_OK;
        }

        __global__ void fold_kernel(ColRef table, Fr r, uint64_t half, Fr* out, bool out_canonical)
        {
            const uint64_t stride = static_cast<uint64_t>(gridDim.x) * blockDim.x;
            // A canonical table enters as stored: r (Montgomery) times a canonical difference is the canonical
            // product, so lo + r (hi - lo) is formed in canonical form and converted once (two
            // multiplications per output instead of three); a Montgomery table needs one, and so does a canonical
            // table folded into a canonical (FR) output: a table that stays in one form costs one per round.
            const bool canonical = deficit(table) != 0;
            for (uint64_t i = static_cast<uint64_t>(blockIdx.x) * blockDim.x + threadIdx.x; i < half; i += stride)
            {
                const Fr lo = col_load_stored(table, 2 * i);
                const Fr hi = col_load_stored(table, 2 * i + 1);
                Fr folded = add(lo, mul(r, sub(hi, lo)));  // in the form of the table
                if (canonical && !out_canonical) folded = to_mont(folded);
                if (!canonical && out_canonical) folded = from_mont(folded);
                store_fr(out + i, folded);
            }
        }

        // Sums of s0 and s1 over the CTA, left with thread 0
        __device__ __forceinline__ void cta_sum_pair(Fr& s0, Fr& s1, Fr* ws0, Fr* ws1)
        {
            const int lane = threadIdx.x & 31;
#pragma unroll 1
            for (int offset = 16; offset > 0; offset >>= 1)
            {
                s0 = add(s0, shfl_fr_idx(s0, (lane + offset) & 31));
                s1 = add(s1, shfl_fr_idx(s1, (lane + offset) & 31));
            }
            if (lane == 0)
            {
                ws0[threadIdx.x >> 5] = s0;
                ws1[threadIdx.x >> 5] = s1;
            }
            __syncthreads();
            if (threadIdx.x < 32)
            {
                s0 = lane < kThreads / 32 ? ws0[lane] : Fr::zero();
                s1 = lane < kThreads / 32 ? ws1[lane] : Fr::zero();
#pragma unroll 1
                for (int offset = kThreads / 64; offset > 0; offset >>= 1)
                {
                    s0 = add(s0, shfl_fr_idx(s0, (lane + offset) & 31));
                    s1 = add(s1, shfl_fr_idx(s1, (lane + offset) & 31));
                }
            }
        }

        // Round sums of a multilinear table for one sumcheck round on a product-free claim:
        // s0 = sum t[2i], s1 = sum t[2i+1].  Every CTA leaves its partial sums; the one that arrives last (nobody
        // waits) adds them up, all its threads together, and writes the result where the host reads it: the
        // rounds of a sumcheck are one short call after another, and a second launch, whose two threads walked
        // through up to 1184 partial sums, took over half of them (all rounds of a 2^20 table: 1697 -> 771 us).
        __global__ void __launch_bounds__(kThreads) round_sums_kernel(ColRef table, uint64_t half, Fr* partial, uint32_t* arrived, Fr* out_canonical)
        {
            __shared__ Fr ws0[kThreads / 32], ws1[kThreads / 32];
            __shared__ bool last;
            Fr s0 = Fr::zero(), s1 = Fr::zero();
            const uint64_t stride = static_cast<uint64_t>(gridDim.x) * blockDim.x;
            // sums of the stored residues; a canonical table stays canonical
            for (uint64_t i = static_cast<uint64_t>(blockIdx.x) * blockDim.x + threadIdx.x; i < half; i += stride)
            {
                s0 = add(s0, col_load_stored(table, 2 * i));
                s1 = add(s1, col_load_stored(table, 2 * i + 1));
            }
            cta_sum_pair(s0, s1, ws0, ws1);
            if (gridDim.x > 1)
            {
                if (threadIdx.x == 0)
                {
                    store_fr(partial + 2 * blockIdx.x, s0);
                    store_fr(partial + 2 * blockIdx.x + 1, s1);
                    __threadfence();
                    last = atomicAdd(arrived, 1u) + 1 == gridDim.x;
                }
                __syncthreads();
                if (!last) return;
                __threadfence();
                s0 = Fr::zero();
                s1 = Fr::zero();
                for (uint32_t b = threadIdx.x; b < gridDim.x; b += kThreads)
                {
                    s0 = add(s0, load_fr_plain(partial + 2 * b));
                    s1 = add(s1, load_fr_plain(partial + 2 * b + 1));
                }
                cta_sum_pair(s0, s1, ws0, ws1);
                if (threadIdx.x == 0) *arrived = 0;  // for the next call
            }
            if (threadIdx.x == 0)
            {
                const bool canonical = deficit(table) != 0;
                store_fr(out_canonical, canonical ? s0 : from_mont(s0));
                store_fr(out_canonical + 1, canonical ? s1 : from_mont(s1));
            }
        }

        int scalar_mont(gzk_ctx* ctx, const uint8_t* bytes, Fr* out)
        {
            bool canonical = false;
            const Fr v = host_fr_from_bytes(bytes, &canonical);
            if (!canonical) return fail(ctx, GZK_E_INVALID, "scalar argument is not a canonical field element");
            *out = to_mont(v);
            return GZK_OK;
        }
    }
}

using namespace gzk;

// The transform behind gzk_ntt and gzk_coset_lde.  `pre`: input i is multiplied by pre^i; `post`: output i by post^i (Montgomery;
// NULL for none); only the first `in_count` elements of each input vector are stored, the others are zeros.
static int ntt_run(gzk_ctx* ctx, const ColRef& in, uint64_t in_count, Fr* out, unsigned log2n, size_t batch, bool inverse, const Fr* pre, const Fr* post)
{
    const uint64_t n = 1ULL << log2n;
    const DomainTables* dom = nullptr;
    int rc = get_domain(ctx, log2n, &dom);
    if (rc != GZK_OK) return rc;

    NttArgs args{};
    args.in = in;
    args.in_count = in_count;
    args.data = out;
    args.lo = inverse ? dom->lo_inv : dom->lo;
    args.hi = inverse ? dom->hi_inv : dom->hi;
    args.lo_bits = dom->lo_bits;
    if ((rc = small_table(ctx, inverse, &args.small)) != GZK_OK) return rc;
    args.log2n = log2n;
    args.scale = dom->inv_size;
    int last_scale_mode = inverse ? 1 : 0;

    if (pre != nullptr || post != nullptr)
    {
        // two-level table of powers of the shift; an inverse transform's 1/n goes into its upper level
        PowerTableArgs powers;
        powers.lo_bits = (log2n + 1) / 2;
        powers.hi_bits = log2n - powers.lo_bits;
        const size_t lo_count = static_cast<size_t>(1) << powers.lo_bits, hi_count = static_cast<size_t>(1) << powers.hi_bits;
        void* scratch = nullptr;
        if ((rc = ensure_scratch(ctx, 2, (lo_count + hi_count) * sizeof(Fr), &scratch)) != GZK_OK) return rc;
        powers.lo = static_cast<Fr*>(scratch);
        powers.hi = powers.lo + lo_count;
        powers.square[0] = pre != nullptr ? *pre : *post;
        for (unsigned k = 1; k < log2n; ++k) powers.square[k] = sqr(powers.square[k - 1]);
        powers.factor = post != nullptr && inverse ? args.scale : Fr::one();
        {
            LaunchScope scope(ctx, "ntt_shift_table");
            power_tables_kernel<<<static_cast<unsigned>((lo_count + hi_count + 127) / 128), 128, 0, ctx->stream>>>(powers);
        }
        GZK_CUDA_TRY(ctx, cudaGetLastError());
        args.shift_lo = powers.lo;
        args.shift_hi = powers.hi;
        args.shift_lo_bits = powers.lo_bits;
        args.pre_shift = pre != nullptr ? 1 : 0;
        if (post != nullptr) last_scale_mode = 2;
    }

    // Pass 0 takes up to 10 stages; the rest is spread evenly over passes of at most 8 stages, each on full
    // 1024-element tiles (2^stages rows of 2^(10-stages) contiguous elements).  A call of fewer tiles than one for
    // every other SM is bound by the length of a tile's chain of rounds, whose butterflies share four schedulers: tiles
    // of 256 elements (8 stages, then at most 6) deal them to four times as many SMs (4 x 2^12 points: 47.9 -> 43.1 us
    // a call, 2^16: 56.6 both ways, 4 x 2^16: 77.7 against 82.6 us).
    bool small_tiles = (n * batch) >> kTileBits < static_cast<uint64_t>(ctx->sm_count) / 2;
#ifdef GZK_BUILD_TUNING
    if (const char* forced = std::getenv("GZK_NTT_SMALL")) small_tiles = std::atoi(forced) != 0;
#endif
    const unsigned tile_bits = small_tiles ? kSmallTileBits : kTileBits;
    const unsigned later = log2n > tile_bits ? log2n - tile_bits : 0;
    const unsigned later_passes = (later + tile_bits - 3) / (tile_bits - 2);
    unsigned later_done = 0, pass_index = 0;
    unsigned s0 = 0;
    do
    {
        const unsigned remaining = log2n - s0;
        unsigned low_bits = 0, stages = 0;
        args.twist = nullptr;
        if (s0 == 0)
        {
            stages = remaining < tile_bits ? remaining : tile_bits;
        }
        else
        {
            // passes still to run share what is left as evenly as possible
            const unsigned passes_left = later_passes - pass_index;
            stages = (later - later_done + passes_left - 1) / passes_left;
            low_bits = tile_bits - stages;
            later_done += stages;
            ++pass_index;
            if ((rc = twist_table(ctx, s0, stages, inverse, &args.twist)) != GZK_OK) return rc;
        }
        args.s0 = s0;
        args.stages = stages;
        args.low_bits = low_bits;
        args.scale_mode = s0 + stages == log2n ? last_scale_mode : 0;
        const unsigned tile_elems = 1u << (stages + low_bits);
        const dim3 grid(static_cast<unsigned>(n / tile_elems), static_cast<unsigned>(batch));
        const unsigned threads = tile_elems >= 4 ? tile_elems / 4 : 1;
        {
            LaunchScope scope(ctx, "ntt_pass");
            if (small_tiles)
                ntt_pass_kernel<kSmallTileBits><<<grid, threads, 0, ctx->stream>>>(args);
            else
                ntt_pass_kernel<kTileBits><<<grid, threads, 0, ctx->stream>>>(args);
        }
        GZK_CUDA_TRY(ctx, cudaGetLastError());
        s0 += stages;
    } while (s0 < log2n);
    return GZK_OK;
}

// A coset shift, in Montgomery form
static int coset_shift_mont(gzk_ctx* ctx, const uint8_t* bytes, Fr* out)
{
    const int rc = scalar_mont(ctx, bytes, out);
    if (rc != GZK_OK) return rc;
    if (out->is_zero()) return fail(ctx, GZK_E_INVALID, "ntt: coset shift must be non-zero");
    return GZK_OK;
}

extern "C"
{
    int gzk_ntt(gzk_ctx* ctx, const gzk_buf* in, gzk_buf* out, unsigned log2n, size_t batch, int inverse, const uint8_t* coset_shift)
    {
        if (ctx == nullptr) return GZK_E_INVALID;
        if (batch == 0) return GZK_OK;
        if (in == nullptr || out == nullptr) return fail(ctx, GZK_E_INVALID, "ntt: null argument");
        if (log2n > 30) return fail(ctx, GZK_E_INVALID, "ntt: domain too large");
        const uint64_t n = 1ULL << log2n;
        if (in->kind == GZK_KIND_F64 || in->kind == GZK_KIND_G1 || in->count < n * batch) return fail(ctx, GZK_E_INVALID, "ntt: input buffer too small or of the wrong kind");
        if (out->kind != GZK_KIND_FR_MONT || out->count < n * batch) return fail(ctx, GZK_E_INVALID, "ntt: output must be a Montgomery buffer of n*batch elements");
        if (out->dptr == in->dptr) return fail(ctx, GZK_E_INVALID, "ntt: input and output must be different buffers");
        if (batch > 65535) return fail(ctx, GZK_E_INVALID, "ntt: batch too large");
        GZK_CUDA_TRY(ctx, cudaSetDevice(ctx->device));
        Fr shift;
        int rc;
        if (coset_shift != nullptr)
        {
            if ((rc = coset_shift_mont(ctx, coset_shift, &shift)) != GZK_OK) return rc;
            if (inverse) shift = inv(shift);
        }
        ColRef column;
        column.ptr = in->dptr;
        column.kind = in->kind;
        rc = ntt_run(ctx, column, n, static_cast<Fr*>(out->dptr), log2n, batch, inverse != 0, coset_shift != nullptr && !inverse ? &shift : nullptr,
                     coset_shift != nullptr && inverse ? &shift : nullptr);
        if (rc != GZK_OK) return rc;
        return wait_call(ctx);
    }

    int gzk_fold(gzk_ctx* ctx, const gzk_buf* table, size_t n, const uint8_t challenge[32], gzk_buf* out)
    {
        if (ctx == nullptr) return GZK_E_INVALID;
        if (n < 2) return GZK_OK;
        if (table == nullptr || out == nullptr || challenge == nullptr) return fail(ctx, GZK_E_INVALID, "fold: null argument");
        if (table->kind == GZK_KIND_F64 || table->kind == GZK_KIND_G1 || table->count < n) return fail(ctx, GZK_E_INVALID, "fold: table buffer too small or of the wrong kind");
        if ((out->kind != GZK_KIND_FR_MONT && out->kind != GZK_KIND_FR) || out->count < n / 2)
            return fail(ctx, GZK_E_INVALID, "fold: output must be an FR or FR_MONT buffer of n/2 elements");
        Fr r;
        int rc = scalar_mont(ctx, challenge, &r);
        if (rc != GZK_OK) return rc;
        GZK_CUDA_TRY(ctx, cudaSetDevice(ctx->device));
        ColRef t;
        t.ptr = table->dptr;
        t.kind = table->kind;
        const uint64_t half = n / 2;
        uint64_t blocks = (half + kThreads - 1) / kThreads;
        const uint64_t cap = static_cast<uint64_t>(ctx->sm_count) * 16;
        if (blocks > cap) blocks = cap;
        {
            LaunchScope scope(ctx, "fold");
            fold_kernel<<<static_cast<unsigned>(blocks), kThreads, 0, ctx->stream>>>(t, r, half, static_cast<Fr*>(out->dptr), out->kind == GZK_KIND_FR);
        }
        GZK_CUDA_TRY(ctx, cudaGetLastError());
        return wait_call(ctx);
    }

    // out[0] = sum_i t[2i], out[1] = sum_i t[2i+1], out[2] = 2*out[1] - out[0]: the values at
    // 0, 1, 2 of the round polynomial sum_i (t[2i] + X (t[2i+1] - t[2i])) of a sumcheck round.
    // With the table split over GPUs each rank computes its three values and the ranks
    // all-gather and add them (gzk_fr_sum) before the Fiat-Shamir squeeze.
    int gzk_sumcheck_round_sums(gzk_ctx* ctx, const gzk_buf* table, size_t n, uint8_t out[3 * 32])
    {
        if (ctx == nullptr) return GZK_E_INVALID;
        if (out == nullptr) return fail(ctx, GZK_E_INVALID, "sumcheck_round_sums: null output");
        std::memset(out, 0, 96);
        if (n < 2) return GZK_OK;
        if (table == nullptr || table->kind == GZK_KIND_F64 || table->kind == GZK_KIND_G1 || table->count < n)
            return fail(ctx, GZK_E_INVALID, "sumcheck_round_sums: table buffer too small or of the wrong kind");
        GZK_CUDA_TRY(ctx, cudaSetDevice(ctx->device));
        const uint64_t half = n / 2;
        uint64_t blocks = (half + kThreads - 1) / kThreads;
        const uint64_t cap = static_cast<uint64_t>(ctx->sm_count) * 4;
        if (blocks > cap) blocks = cap;
        void* scratch = nullptr;
        void* result = nullptr;
        int rc = ensure_scratch(ctx, 2, 2 * blocks * sizeof(Fr), &scratch);
        if (rc == GZK_OK) rc = ensure_pinned(ctx, 2 * sizeof(Fr), &result);
        if (rc != GZK_OK) return rc;
        Fr* partial = static_cast<Fr*>(scratch);
        ColRef t;
        t.ptr = table->dptr;
        t.kind = table->kind;
        {
            LaunchScope scope(ctx, "round_sums");
            round_sums_kernel<<<static_cast<unsigned>(blocks), kThreads, 0, ctx->stream>>>(t, half, partial, ctx->arrival_counter(), static_cast<Fr*>(result));
        }
        GZK_CUDA_TRY(ctx, cudaGetLastError());
        GZK_CUDA_TRY(ctx, cudaStreamSynchronize(ctx->stream));
        std::memcpy(out, result, 64);
        // value at 2 = s0 + 2 (s1 - s0) = 2 s1 - s0, on the host
        uint8_t twice[32];
        if (gzk_fr_op(0, out + 32, out + 32, twice) != GZK_OK || gzk_fr_op(1, twice, out, out + 64) != GZK_OK)
            return fail(ctx, GZK_E_INVALID, "sumcheck_round_sums: internal arithmetic error");
        return GZK_OK;
    }

    // Coset low-degree extension: evaluations on the 2^log2n domain -> evaluations of the
    // same polynomial on shift * (2^(log2n+log2_blowup) domain).
    int gzk_coset_lde(gzk_ctx* ctx, const gzk_buf* in, unsigned log2n, unsigned log2_blowup, const uint8_t shift[32], gzk_buf* out)
    {
        if (ctx == nullptr) return GZK_E_INVALID;
        if (in == nullptr || out == nullptr || shift == nullptr) return fail(ctx, GZK_E_INVALID, "coset_lde: null argument");
        if (log2n + log2_blowup > 30) return fail(ctx, GZK_E_INVALID, "coset_lde: extended domain too large");
        const size_t n = static_cast<size_t>(1) << log2n, big = n << log2_blowup;
        if (out->kind != GZK_KIND_FR_MONT || out->count < big) return fail(ctx, GZK_E_INVALID, "coset_lde: output must be a Montgomery buffer of the extended size");
        if (in->kind == GZK_KIND_F64 || in->kind == GZK_KIND_G1 || in->count < n) return fail(ctx, GZK_E_INVALID, "ntt: input buffer too small or of the wrong kind");
        GZK_CUDA_TRY(ctx, cudaSetDevice(ctx->device));
        Fr g;
        int rc = coset_shift_mont(ctx, shift, &g);
        if (rc != GZK_OK) return rc;
        // The n coefficients, already times shift^i, lie in the context's scratch; an allocation per call and its release
        // (14.7 ms a call in a row of them at 2^20) only where they would tie up more than kKeptCoefficients.
        constexpr size_t kKeptCoefficients = static_cast<size_t>(256) << 20;
        gzk_buf* own = nullptr;
        void* coefficients = nullptr;
        if (n * sizeof(Fr) <= kKeptCoefficients)
        {
            rc = ensure_scratch(ctx, 1, n * sizeof(Fr), &coefficients);
        }
        else if ((rc = gzk_buf_alloc(ctx, GZK_KIND_FR_MONT, n, &own)) == GZK_OK)
        {
            coefficients = own->dptr;
        }
        if (rc != GZK_OK) return rc;
        ColRef column;
        column.ptr = in->dptr;
        column.kind = in->kind;
        rc = ntt_run(ctx, column, n, static_cast<Fr*>(coefficients), log2n, 1, true, nullptr, &g);
        column.ptr = coefficients;
        column.kind = GZK_KIND_FR_MONT;
        // the coefficients beyond the n-th are zeros that are never stored
        if (rc == GZK_OK) rc = ntt_run(ctx, column, n, static_cast<Fr*>(out->dptr), log2n + log2_blowup, 1, false, nullptr, nullptr);
        if (rc == GZK_OK) rc = wait_call(ctx);
        if (own == nullptr) return rc;
        const std::string message = ctx->last_error;
        gzk_buf_free(ctx, own);
        if (rc != GZK_OK) ctx->last_error = message;
        return rc;
    }
}
