// G1 multi-scalar multiplication sum_i [s_i] P_i by the bucket (Pippenger) method
// with signed-digit windows and XYZZ bucket accumulators.
//
//   1. digits     every scalar is cut into W signed c-bit digits; per (window, |digit|)
//                 bucket the number of hits is counted
//   2. offsets    exclusive scan of the bucket counts (one CTA)
//   3. scatter    (point index, sign) pairs are written bucket by bucket
//   4. buckets    one to eight lanes per bucket, longest buckets first, add its points (mixed XYZZ additions)
//   5. bits       sum_d d*B_d of a bucket set: row and column sums of the buckets laid out as a
//                 matrix, then the two small weighted sums split by the bits of the multiplier
//   6. windows    sum of 2^b times the sums of the bits, a quad of lanes per bit; the host shifts the window
//                 sums by 2^(c*w), adds them and converts to affine (254 dependent doublings: 0.2 ms there,
//                 1.8 ms as a chain of one GPU thread)
//
// With a precomputed table of the points shifted by every window (gzk_msm_precompute:
// 2^(c*w) P_i for all w, the layout for a resident SRS) the digits of all windows fall
// into ONE set of 2^(c-1) buckets: no per-window reduction and no chain of c*w doublings
// at the end, and the window can
// be wider because only one window's buckets are reduced.
//
// Signed digits halve the bucket count (2^(c-1) per window): a negative digit adds
// the negated point.  Group sums do not depend on the order of additions, so the
// atomics of steps 1 and 3 leave the result bit-identical from run to run.
#include <cstdlib>
#include <cstring>
#include <vector>

#include "block.cuh"
#include "g1.cuh"
#include "g1_quad.cuh"
#include "host_g1.hpp"

namespace gzk
{
    namespace
    {
        constexpr int kThreads = 128;
        constexpr int kMaxWindows = 32;
        // Buckets with more than four times the mean of their plan (`big`; skewed scalars: small integers, constant
        // columns, the short top window) are cut into slices; one CTA sums a slice, one CTA then adds the
        // slices of a bucket.  Short slices make the chains short (a thread adds four points of a slice of
        // 512, and a quad of lanes joins them), and a very long bucket has at most 256.
        constexpr uint32_t kBigBucketMin = 128, kBigBucketMax = 1024;
        constexpr uint32_t kSliceEntries = 512;
        constexpr uint32_t kMaxSlices = 256;
        __device__ __forceinline__ uint32_t slice_entries(uint32_t size)
        {
            const uint32_t even = (size + kMaxSlices - 1) / kMaxSlices;
            return even > kSliceEntries ? even : kSliceEntries;
        }

        struct BigItem
        {
            uint32_t bucket;
            uint32_t slice;
        };
        struct BigBucket
        {
            uint32_t bucket;
            uint32_t first_item;
            uint32_t slices;
        };

        struct MsmPlan
        {
            uint32_t c;        // window bits
            uint32_t windows;  // ceil(256 / c)
            uint32_t half;     // 2^(c-1) buckets per window
            uint32_t shared;   // 1: all windows share one bucket set and entries index the shifted-point table [w*n + i]
        };

        // code[w*n + i] = 0 for a zero digit, else ((|d|-1) << 1 | negative) + 1
        __global__ void __launch_bounds__(kThreads) msm_digits_kernel(ColRef scalars, uint64_t n, MsmPlan plan, uint32_t* code,
                                                                     uint32_t* bucket_count)
        {
            const uint64_t i = static_cast<uint64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
            if (i >= n) return;
            Fr s = load_fr(static_cast<const Fr*>(scalars.ptr) + i);
            if (scalars.kind == GZK_KIND_FR_MONT) s = from_mont(s);
            uint32_t carry = 0;
            for (uint32_t w = 0; w < plan.windows; ++w)
            {
                const uint32_t bit = w * plan.c;
                uint32_t raw = 0;
                if (bit < 256)
                {
                    const uint32_t limb = bit >> 5, shift = bit & 31;
                    uint64_t two = s.l[limb];
                    if (limb + 1 < 8) two |= static_cast<uint64_t>(s.l[limb + 1]) << 32;
                    raw = static_cast<uint32_t>(two >> shift) & ((1u << plan.c) - 1u);
                }
                uint32_t d = raw + carry;
                uint32_t negative = 0;
                carry = 0;
                if (d > plan.half)
                {
                    d = (1u << plan.c) - d;
                    negative = 1;
                    carry = 1;
                }
                uint32_t out = 0;
                if (d != 0)
                {
                    out = (((d - 1) << 1) | negative) + 1;
                    atomicAdd(bucket_count + (plan.shared ? 0 : static_cast<uint64_t>(w) * plan.half) + (d - 1), 1u);
                }
                code[static_cast<uint64_t>(w) * n + i] = out;
            }
        }

        // start = exclusive scan of `count` sizes by one CTA; also zeroes `cursor`.  Eight values per thread and round:
        // the rounds follow one another, and with one value each the 2^16 buckets of a table took 71 us.
        constexpr uint32_t kScanElems = 8;
        __global__ void __launch_bounds__(1024) msm_offsets_kernel(const uint32_t* sizes, uint32_t* start, uint32_t* cursor, uint32_t count)
        {
            __shared__ uint32_t warp_totals[32];
            const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
            uint32_t carry = 0;
            for (uint32_t base = 0; base < count; base += 1024 * kScanElems)
            {
                const uint32_t first = base + threadIdx.x * kScanElems;
                uint32_t v[kScanElems], sum = 0;
#pragma unroll
                for (uint32_t j = 0; j < kScanElems; ++j)
                {
                    v[j] = first + j < count ? sizes[first + j] : 0;
                    sum += v[j];
                }
                uint32_t incl = sum;
#pragma unroll
                for (int offset = 1; offset < 32; offset <<= 1)
                {
                    const uint32_t up = __shfl_up_sync(0xffffffffu, incl, offset);
                    if (lane >= static_cast<uint32_t>(offset)) incl += up;
                }
                if (lane == 31) warp_totals[warp] = incl;
                __syncthreads();
                uint32_t totals = warp_totals[lane];
#pragma unroll
                for (int offset = 1; offset < 32; offset <<= 1)
                {
                    const uint32_t up = __shfl_up_sync(0xffffffffu, totals, offset);
                    if (lane >= static_cast<uint32_t>(offset)) totals += up;
                }
                const uint32_t before = __shfl_sync(0xffffffffu, totals, (warp + 31) & 31);
                uint32_t run = carry + (warp == 0 ? 0 : before) + incl - sum;
#pragma unroll
                for (uint32_t j = 0; j < kScanElems; ++j)
                {
                    if (first + j < count)
                    {
                        start[first + j] = run;
                        cursor[first + j] = 0;
                    }
                    run += v[j];
                }
                carry += __shfl_sync(0xffffffffu, totals, 31);
                __syncthreads();
            }
        }

        // The buckets by size, longest first: the lanes of a warp then add equally many points (bucket sizes scatter
        // by their square root, so that the longest of 32 holds a fifth more than the mean at 240 points and two
        // thirds more at 16), and the last warps to start have the least to do.  Buckets the slices take come last,
        // with size 0.
        constexpr uint32_t kSizeBins = kBigBucketMax + 1;
        __device__ __forceinline__ uint32_t size_bin(uint32_t size, uint32_t big) { return size > big ? kBigBucketMax : kBigBucketMax - size; }
        __global__ void __launch_bounds__(1024) msm_size_histogram_kernel(const uint32_t* bucket_size, uint32_t buckets, uint32_t big, uint32_t* histogram)
        {
            __shared__ uint32_t local[kSizeBins];
            for (uint32_t i = threadIdx.x; i < kSizeBins; i += blockDim.x) local[i] = 0;
            __syncthreads();
            const uint32_t b = blockIdx.x * blockDim.x + threadIdx.x;
            if (b < buckets) atomicAdd(local + size_bin(bucket_size[b], big), 1u);
            __syncthreads();
            for (uint32_t i = threadIdx.x; i < kSizeBins; i += blockDim.x)
                if (local[i] != 0) atomicAdd(histogram + i, local[i]);
        }
        // `cursor`: one zeroed word per bin
        __global__ void __launch_bounds__(1024) msm_order_kernel(const uint32_t* bucket_size, uint32_t buckets, uint32_t big, const uint32_t* histogram, uint32_t* cursor, uint32_t* order)
        {
            __shared__ uint32_t first[kSizeBins], local[kSizeBins];
            __shared__ uint32_t warp_totals[32];
            static_assert(kSizeBins == 1025, "one bin per thread, the last one at the end");
            const uint32_t t = threadIdx.x, lane = t & 31, warp = t >> 5;
            const uint32_t v = histogram[t];
            uint32_t incl = v;
#pragma unroll
            for (int offset = 1; offset < 32; offset <<= 1)
            {
                const uint32_t up = __shfl_up_sync(0xffffffffu, incl, offset);
                if (lane >= static_cast<uint32_t>(offset)) incl += up;
            }
            if (lane == 31) warp_totals[warp] = incl;
            local[t] = 0;
            if (t == 0) local[1024] = 0;
            __syncthreads();
            uint32_t before = 0;
            for (uint32_t w = 0; w < warp; ++w) before += warp_totals[w];
            first[t] = before + incl - v;
            if (t == 1023) first[1024] = before + incl;
            __syncthreads();
            const uint32_t b = blockIdx.x * blockDim.x + t;
            uint32_t bin = 0, rank = 0;
            if (b < buckets)
            {
                bin = size_bin(bucket_size[b], big);
                rank = atomicAdd(local + bin, 1u);
            }
            __syncthreads();
            for (uint32_t i = t; i < kSizeBins; i += 1024)
                if (local[i] != 0) first[i] += atomicAdd(cursor + i, local[i]);
            __syncthreads();
            if (b < buckets) order[first[bin] + rank] = b;
        }

        __global__ void __launch_bounds__(kThreads) msm_scatter_kernel(const uint32_t* code, uint64_t n, MsmPlan plan,
                                                                      const uint32_t* bucket_start, uint32_t* cursor, uint32_t* entries)
        {
            const uint64_t total = n * plan.windows;
            const uint64_t stride = static_cast<uint64_t>(gridDim.x) * blockDim.x;
            for (uint64_t t = static_cast<uint64_t>(blockIdx.x) * blockDim.x + threadIdx.x; t < total; t += stride)
            {
                const uint32_t v = code[t];
                if (v == 0) continue;
                const uint64_t w = t / n;
                const uint64_t i = t - w * n;
                const uint32_t payload = v - 1;
                const uint64_t bucket = (plan.shared ? 0 : w * plan.half) + (payload >> 1);
                const uint32_t pos = atomicAdd(cursor + bucket, 1u);
                entries[bucket_start[bucket] + pos] = (static_cast<uint32_t>(plan.shared ? t : i) << 1) | (payload & 1u);
            }
        }

        template <int WIDTH>
        __device__ __forceinline__ G1Xyzz shfl_down_xyzz(const G1Xyzz& p, int offset)
        {
            G1Xyzz o;
#pragma unroll
            for (int i = 0; i < FpCfg::N; ++i)
            {
                o.X.l[i] = __shfl_down_sync(0xffffffffu, p.X.l[i], offset, WIDTH);
                o.Y.l[i] = __shfl_down_sync(0xffffffffu, p.Y.l[i], offset, WIDTH);
                o.ZZ.l[i] = __shfl_down_sync(0xffffffffu, p.ZZ.l[i], offset, WIDTH);
                o.ZZZ.l[i] = __shfl_down_sync(0xffffffffu, p.ZZZ.l[i], offset, WIDTH);
            }
            return o;
        }

        // LANES adjacent lanes per bucket, buckets in the order of their sizes
        template <int LANES>
        __global__ void __launch_bounds__(kThreads) msm_buckets_kernel(const G1Affine* points, const uint32_t* bucket_start,
                                                                      const uint32_t* bucket_size, const uint32_t* order, const uint32_t* entries,
                                                                      uint32_t buckets, uint32_t big, G1Xyzz* out)
        {
            const uint32_t t = blockIdx.x * blockDim.x + threadIdx.x;
            const uint32_t slot = t / LANES, part = t % LANES;
            const uint32_t b = slot < buckets ? order[slot] : 0;
            const uint32_t start = bucket_start[b], size = slot < buckets ? bucket_size[b] : 0;
            const bool mine = size <= big;  // longer ones are handled cooperatively by msm_big_slices_kernel
            G1Xyzz acc = G1Xyzz::infinity();
            if (mine)
            {
#pragma unroll 1
                for (uint32_t k = part; k < size; k += LANES)
                {
                    const uint32_t e = entries[start + k];
                    acc = g1_add_mixed(acc, load_affine(points + (e >> 1)), (e & 1u) != 0);
                }
            }
#pragma unroll 1
            for (int offset = LANES / 2; offset > 0; offset >>= 1)
            {
                const G1Xyzz other = shfl_down_xyzz<LANES>(acc, offset);
                if (part < static_cast<uint32_t>(offset)) acc = g1_add(acc, other);
            }
            if (mine && part == 0 && slot < buckets) store_xyzz(out + b, acc);
        }

        // counters[0] = number of slice items, counters[1] = number of big buckets
        __global__ void __launch_bounds__(kThreads) msm_plan_big_kernel(const uint32_t* bucket_size, uint32_t buckets, uint32_t threshold, uint32_t* counters,
                                                                       BigItem* items, BigBucket* big)
        {
            const uint32_t b = blockIdx.x * blockDim.x + threadIdx.x;
            if (b >= buckets) return;
            const uint32_t size = bucket_size[b];
            if (size <= threshold) return;
            const uint32_t entries = slice_entries(size), slices = (size + entries - 1) / entries;
            const uint32_t first = atomicAdd(counters, slices);
            const uint32_t slot = atomicAdd(counters + 1, 1u);
            BigBucket bb;
            bb.bucket = b;
            bb.first_item = first;
            bb.slices = slices;
            big[slot] = bb;
            for (uint32_t j = 0; j < slices; ++j)
            {
                BigItem it;
                it.bucket = b;
                it.slice = j;
                items[first + j] = it;
            }
        }

        // Sum over the 32 quads of a CTA of 128 threads, returned to quad 0
        __device__ __forceinline__ Fp quad_cta_sum(Fp p, Fp* slots /* 16 */)
        {
            static_assert(kThreads == 128, "four warps of eight quads");
#pragma unroll 1
            for (int mask = 4; mask <= 64; mask <<= 1)
            {
                if (mask == 32)
                {
                    if ((threadIdx.x & 31) < 4) slots[(threadIdx.x >> 5) * 4 + (threadIdx.x & 3)] = p;
                    __syncthreads();
                    p = slots[threadIdx.x & 15];
                }
                p = quad_add(p, shfl_xor_fp(p, mask < 32 ? mask : mask >> 3));
            }
            return p;
        }
        // Slice items dealt to the CTAs: the threads stride over a slice, then the quads add the threads' sums up
        // (four multiplications deep per addition: 258 -> 72 of them in sequence for a slice)
        __global__ void __launch_bounds__(kThreads) msm_big_slices_kernel(const G1Affine* points, const uint32_t* bucket_start,
                                                                         const uint32_t* bucket_size, const uint32_t* entries,
                                                                         const uint32_t* counters, const BigItem* items, G1Xyzz* partial)
        {
            __shared__ G1Xyzz sums[kThreads];
            __shared__ Fp slots[16];
            const uint32_t quad = threadIdx.x >> 2, role = threadIdx.x & 3, count = counters[0];
            for (uint32_t item = blockIdx.x; item < count; item += gridDim.x)
            {
                const BigItem it = items[item];
                const uint32_t start = bucket_start[it.bucket], size = bucket_size[it.bucket], length = slice_entries(size);
                const uint32_t begin = it.slice * length;
                const uint32_t end = begin + length < size ? begin + length : size;
                G1Xyzz acc = G1Xyzz::infinity();
#pragma unroll 1
                for (uint32_t k = begin + threadIdx.x; k < end; k += kThreads)
                {
                    const uint32_t e = entries[start + k];
                    acc = g1_add_mixed(acc, load_affine(points + (e >> 1)), (e & 1u) != 0);
                }
                sums[threadIdx.x] = acc;
                __syncthreads();
                const Fp* parts = reinterpret_cast<const Fp*>(sums);
                Fp p = parts[4 * quad + role];
#pragma unroll 1
                for (uint32_t j = 1; j < 4; ++j) p = quad_add(p, parts[4 * (quad + 32 * j) + role]);
                p = quad_cta_sum(p, slots);
                if (threadIdx.x < 4) store_fp(reinterpret_cast<Fp*>(partial + item) + role, p);
                __syncthreads();
            }
        }

        // CTA per big bucket: the quads stride over its slice sums, then a tree
        __global__ void __launch_bounds__(kThreads) msm_big_combine_kernel(const uint32_t* counters, const BigBucket* big, const G1Xyzz* partial,
                                                                          G1Xyzz* out)
        {
            __shared__ Fp slots[16];
            const uint32_t quad = threadIdx.x >> 2, role = threadIdx.x & 3, count = counters[1];
            for (uint32_t item = blockIdx.x; item < count; item += gridDim.x)
            {
                const BigBucket bb = big[item];
                const Fp* parts = reinterpret_cast<const Fp*>(partial + bb.first_item);
                Fp p = Fp::zero();
#pragma unroll 1
                for (uint32_t base = 0; base < bb.slices; base += kThreads / 4)
                {
                    const uint32_t j = base + quad;
                    Fp q = Fp::zero();
                    if (j < bb.slices) q = parts[4 * static_cast<size_t>(j) + role];
                    p = base == 0 ? q : quad_add(p, q);
                }
                p = quad_cta_sum(p, slots);
                if (threadIdx.x < 4) store_fp(reinterpret_cast<Fp*>(out + bb.bucket) + role, p);
                __syncthreads();
            }
        }

        // ---- shared-bucket path: reduction of ONE bucket set -----------------------------------
        // sum_d d * B_d over d = 1 .. 2^(c-1) (B_d = bucket d-1).  Write d = hi * 2^h + lo and lay the
        // buckets out as a matrix [hi][lo]: with the row sums R_hi and the column sums C_lo,
        //   sum_d d * B_d = sum_lo lo * C_lo + 2^h * sum_hi hi * R_hi,
        // so the bulk of the work is 2 additions per bucket in short independent trees, and the
        // two weighted sums run over 2^h and 2^(c-1-h)+1 points only; those are split by the bits
        // of the multiplier: bit_sums[b] for b < h from the columns, for b >= h from the rows,
        // and sum_b 2^b * bit_sums[b] is the result.
        // LANES adjacent lanes per line: lines [0, rows) are rows, lines [rows, rows + cols) columns.  rc = [rows row
        // sums][cols column sums] (blockIdx.y = window when every window has its own bucket set)
        template <int LANES>
        __global__ void __launch_bounds__(kThreads) msm_rowcol_kernel(const G1Xyzz* buckets, uint32_t half, uint32_t h, uint32_t rows, G1Xyzz* rc)
        {
            const uint32_t cols = 1u << h, t = blockIdx.x * kThreads + threadIdx.x, line = t / LANES, part = t % LANES;
            buckets += static_cast<uint64_t>(blockIdx.y) * half;
            rc += static_cast<uint64_t>(blockIdx.y) * (rows + cols);
            // d = first + k * step for k < length, of which 1 .. half are buckets
            const bool row = line < rows;
            const uint32_t first = row ? line << h : line - rows, step = row ? 1u : cols, length = line >= rows + cols ? 0u : row ? cols : rows;
            G1Xyzz acc = G1Xyzz::infinity();
#pragma unroll 1
            for (uint32_t k = part; k < length; k += LANES)
            {
                const uint32_t d = first + k * step;
                if (d >= 1 && d <= half) acc = g1_add(acc, load_xyzz(buckets + (d - 1)));
            }
#pragma unroll 1
            for (int offset = LANES / 2; offset > 0; offset >>= 1)
            {
                const G1Xyzz other = shfl_down_xyzz<LANES>(acc, offset);
                if (part < static_cast<uint32_t>(offset)) acc = g1_add(acc, other);
            }
            if (part == 0 && line < rows + cols) store_xyzz(rc + line, acc);
        }

        // CTA b < h: sum of the column sums whose lo has bit b; CTA b >= h: sum of the row sums whose hi has bit b - h
        __global__ void __launch_bounds__(kThreads) msm_rowcol_bits_kernel(const G1Xyzz* rc, uint32_t h, uint32_t rows, G1Xyzz* bit_sums)
        {
            __shared__ Fp slots[16];
            const uint32_t b = blockIdx.x, quad = threadIdx.x >> 2, role = threadIdx.x & 3;
            rc += static_cast<uint64_t>(blockIdx.y) * (rows + (1u << h));
            bit_sums += static_cast<uint64_t>(blockIdx.y) * gridDim.x;
            const bool from_cols = b < h;
            const uint32_t count = from_cols ? (1u << h) : rows;
            const uint32_t bit = from_cols ? b : b - h;
            const Fp* src = reinterpret_cast<const Fp*>(from_cols ? rc + rows : rc);
            Fp acc = Fp::zero();
#pragma unroll 1
            for (uint32_t base = 0; base < (count + 1) / 2; base += kThreads / 4)
            {
                const uint32_t i = base + quad;  // the i-th number with that bit set
                const uint32_t j = (i >> bit) << (bit + 1) | 1u << bit | (i & ((1u << bit) - 1u));
                Fp p = Fp::zero();
                if (j < count) p = src[4 * static_cast<size_t>(j) + role];
                acc = base == 0 ? p : quad_add(acc, p);
            }
            acc = quad_cta_sum(acc, slots);
            if (threadIdx.x < 4) store_fp(reinterpret_cast<Fp*>(bit_sums + b) + role, acc);
        }
        // CTA per bucket set: quad b doubles the sum of bit b by b times, then a tree
        __global__ void __launch_bounds__(kThreads) msm_window_sums_kernel(const G1Xyzz* bit_sums, uint32_t c, G1Xyzz* out)
        {
            __shared__ Fp slots[16];
            const uint32_t b = threadIdx.x >> 2, role = threadIdx.x & 3;
            bit_sums += static_cast<uint64_t>(blockIdx.x) * c;
            Fp p = Fp::zero();
            if (b < c) p = reinterpret_cast<const Fp*>(bit_sums)[4 * b + role];
#pragma unroll 1
            for (uint32_t k = 0; k + 1 < c; ++k)
            {
                const Fp twice = quad_double(p);
                if (k < b) p = twice;
            }
            p = quad_cta_sum(p, slots);
            if (threadIdx.x < 4) store_fp(reinterpret_cast<Fp*>(out + blockIdx.x) + role, p);
        }

        // next[i] = 2^c * prev[i] (affine Montgomery in and out; one inversion per point, all in parallel)
        __global__ void __launch_bounds__(kThreads) msm_table_window_kernel(const G1Affine* prev, G1Affine* next, uint64_t n, uint32_t c)
        {
            const uint64_t i = static_cast<uint64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
            if (i >= n) return;
            const G1Affine p = load_affine(prev + i);
            if (p.is_infinity())
            {
                store_affine(next + i, p);
                return;
            }
            G1Xyzz acc = G1Xyzz::from_affine(p);
#pragma unroll 1
            for (uint32_t k = 0; k < c; ++k) acc = g1_double(acc);
            store_affine(next + i, g1_to_affine(acc));
        }

        // Windows needed for scalars below the group order r: ceil(255 / c), plus one when the top
        // digit could still reach 2^(c-1) and push a carry out.
        uint32_t windows_for(uint32_t c)
        {
            uint32_t windows = (255 + c - 1) / c;
            const uint32_t top_shift = c * (windows - 1);
            // largest top digit = (r - 1) >> top_shift, from the modulus limbs
            uint64_t top = 0;
            for (int limb = 7; limb >= 0; --limb)
            {
                const uint32_t lo_bit = 32u * static_cast<uint32_t>(limb);
                if (lo_bit + 32 <= top_shift) break;
                const uint64_t word = FrCfg::mod(limb);
                if (lo_bit >= top_shift)
                    top |= word << (lo_bit - top_shift);
                else
                    top |= word >> (top_shift - lo_bit);
            }
            if (top + 1 > (1ULL << (c - 1))) ++windows;  // top digit + incoming carry may exceed the signed range
            return windows;
        }

        MsmPlan make_shared_plan(uint32_t c)
        {
            MsmPlan p;
            p.c = c;
            p.windows = windows_for(c);
            p.half = 1u << (c - 1);
            p.shared = 1;
            return p;
        }

        // Window of a plan with a bucket set per window, by multiplications: ten per point and window, about 45 per
        // bucket for its two additions in the row and column sums, and half a window again where the top window has
        // so few bits that its handful of buckets goes through the slices.
        int plan_window_bits(uint64_t n)
        {
            int best = 8;
            double best_cost = 0.0;
            for (int c = 8; c <= 16; ++c)
            {
                const int windows = (256 + c - 1) / c, top_bits = 255 - c * (windows - 1);
                double cost = 10.0 * static_cast<double>(n) * windows + 45.0 * windows * static_cast<double>(1u << (c - 1));
                if (top_bits < c - 3) cost += 5.0 * static_cast<double>(n);
                if (best_cost == 0.0 || cost < best_cost)
                {
                    best_cost = cost;
                    best = c;
                }
            }
            return best;
        }

        // Lanes per bucket: two points for every lane until each scheduler has four warps, sixteen until it has
        // sixteen (more warps even out the last wave; joining the lanes costs as much as 1.4 points a level).  One
        // lane per bucket left 13312 lanes for 2^16 points: bucket pass 1773 us, with window and lanes chosen as here
        // 662 us (whole call 5.27 -> 1.37 ms).  2^20 points on their table, 240 to a bucket: call 8.43 / 7.74 / 7.44 ms
        // with 1 / 2 / 4 lanes (9.36 ms before the buckets were ordered).
        uint32_t bucket_lanes(const gzk_ctx* ctx, uint64_t buckets, uint64_t entries)
        {
            const uint64_t four_warps = static_cast<uint64_t>(ctx->sm_count) * 4 * 4 * 32;
            uint32_t lanes = 1;
            while (lanes < 8 && buckets * lanes * 2 <= (entries >= buckets * lanes * 32 ? 4 * four_warps : four_warps) && entries >= buckets * lanes * 4) lanes *= 2;
#ifdef GZK_BUILD_TUNING
            if (const char* forced = std::getenv("GZK_MSM_LANES")) lanes = static_cast<uint32_t>(std::atoi(forced));
#endif
            return lanes;
        }

        MsmPlan make_plan(uint64_t n)
        {
            int c = plan_window_bits(n);
#ifdef GZK_BUILD_TUNING
            if (const char* forced = std::getenv("GZK_MSM_WINDOW")) c = std::atoi(forced);
#endif
            MsmPlan p;
            p.c = static_cast<uint32_t>(c);
            p.windows = (256 + p.c - 1) / p.c;
            p.half = 1u << (p.c - 1);
            p.shared = 0;
            return p;
        }
    }

    // MSM over device-resident scalars and points; the canonical affine result is written to `out_host`.
    static int msm_run_plan(gzk_ctx* ctx, const gzk_buf* scalars, const gzk_buf* points, uint64_t n, const MsmPlan& plan, uint8_t out_host[96])
    {
        const uint64_t buckets = plan.shared ? plan.half : static_cast<uint64_t>(plan.windows) * plan.half;
        const size_t code_bytes = static_cast<size_t>(n) * plan.windows * sizeof(uint32_t);
        const size_t bucket_u32 = buckets * sizeof(uint32_t);
        const uint64_t total_entries = n * plan.windows;
        const uint64_t four_means = 4 * total_entries / buckets;
        const uint32_t big = four_means < kBigBucketMin ? kBigBucketMin : four_means > kBigBucketMax ? kBigBucketMax : static_cast<uint32_t>(four_means);
        const uint64_t max_big = total_entries / big + 1;          // buckets that can exceed the threshold
        const uint64_t max_items = total_entries / kSliceEntries + max_big; // sum of ceil(size / slice) over them
        const size_t big_bytes = max_items * (sizeof(BigItem) + sizeof(G1Xyzz)) + max_big * sizeof(BigBucket) + 64;
        const uint32_t split_h = (plan.c - 1) / 2;                          // low bits of the bucket multiplier
        const uint32_t split_rows = (1u << (plan.c - 1 - split_h)) + 1;     // values of the high part, 0 .. 2^(c-1-h)
        const uint32_t bucket_sets = plan.shared ? 1u : plan.windows;
        const size_t chunk_bytes = static_cast<size_t>(bucket_sets) * (static_cast<size_t>(split_rows) + (1u << split_h)) * sizeof(G1Xyzz);
        const size_t total = big_bytes + 2 * code_bytes + 3 * bucket_u32 + buckets * sizeof(G1Xyzz) + static_cast<size_t>(plan.windows) * plan.c * sizeof(G1Xyzz) +
                             chunk_bytes + static_cast<size_t>(plan.windows) * sizeof(G1Xyzz) + bucket_u32 + 2 * kSizeBins * sizeof(uint32_t) + 8192;
        void* scratch = nullptr;
        int rc = ensure_scratch(ctx, 1, total, &scratch);
        if (rc != GZK_OK) return rc;
        char* cur = static_cast<char*>(scratch);
        auto take = [&](size_t bytes) {
            char* p = cur;
            cur += (bytes + 255) & ~static_cast<size_t>(255);
            return p;
        };
        G1Xyzz* bucket_points = reinterpret_cast<G1Xyzz*>(take(buckets * sizeof(G1Xyzz)));
        G1Xyzz* bit_sums = reinterpret_cast<G1Xyzz*>(take(static_cast<size_t>(plan.windows) * plan.c * sizeof(G1Xyzz)));
        G1Xyzz* window_sums = reinterpret_cast<G1Xyzz*>(take(static_cast<size_t>(plan.windows) * sizeof(G1Xyzz)));
        uint32_t* order = reinterpret_cast<uint32_t*>(take(bucket_u32));
        uint32_t* size_bins = reinterpret_cast<uint32_t*>(take(2 * kSizeBins * sizeof(uint32_t)));
        uint32_t* code = reinterpret_cast<uint32_t*>(take(code_bytes));
        uint32_t* entries = reinterpret_cast<uint32_t*>(take(code_bytes));
        uint32_t* bucket_size = reinterpret_cast<uint32_t*>(take(bucket_u32));
        uint32_t* bucket_start = reinterpret_cast<uint32_t*>(take(bucket_u32));
        uint32_t* cursor = reinterpret_cast<uint32_t*>(take(bucket_u32));
        G1Xyzz* big_partial = reinterpret_cast<G1Xyzz*>(take(max_items * sizeof(G1Xyzz)));
        BigItem* big_items = reinterpret_cast<BigItem*>(take(max_items * sizeof(BigItem)));
        BigBucket* big_buckets = reinterpret_cast<BigBucket*>(take(max_big * sizeof(BigBucket)));
        uint32_t* big_counters = reinterpret_cast<uint32_t*>(take(64));
        G1Xyzz* bit_partial = reinterpret_cast<G1Xyzz*>(take(chunk_bytes));
        if (static_cast<size_t>(cur - static_cast<char*>(scratch)) > ctx->scratch[1].bytes)
            return fail(ctx, GZK_E_INVALID, "msm: internal scratch accounting error");

        ColRef s;
        s.ptr = scalars->dptr;
        s.kind = scalars->kind;
        GZK_CUDA_TRY(ctx, cudaMemsetAsync(bucket_size, 0, bucket_u32, ctx->stream));
        {
            LaunchScope scope(ctx, "msm_digits");
            msm_digits_kernel<<<static_cast<unsigned>((n + kThreads - 1) / kThreads), kThreads, 0, ctx->stream>>>(s, n, plan, code, bucket_size);
        }
        GZK_CUDA_TRY(ctx, cudaGetLastError());
        {
            LaunchScope scope(ctx, "msm_offsets");
            msm_offsets_kernel<<<1, 1024, 0, ctx->stream>>>(bucket_size, bucket_start, cursor, static_cast<uint32_t>(buckets));
        }
        GZK_CUDA_TRY(ctx, cudaGetLastError());
        {
            LaunchScope scope(ctx, "msm_scatter");
            const uint64_t work = n * plan.windows;
            uint64_t blocks = (work + kThreads - 1) / kThreads;
            const uint64_t cap = static_cast<uint64_t>(ctx->sm_count) * 32;
            if (blocks > cap) blocks = cap;
            msm_scatter_kernel<<<static_cast<unsigned>(blocks), kThreads, 0, ctx->stream>>>(code, n, plan, bucket_start, cursor, entries);
        }
        GZK_CUDA_TRY(ctx, cudaGetLastError());
        GZK_CUDA_TRY(ctx, cudaMemsetAsync(big_counters, 0, 64, ctx->stream));
        {
            LaunchScope scope(ctx, "msm_plan_big");
            msm_plan_big_kernel<<<static_cast<unsigned>((buckets + kThreads - 1) / kThreads), kThreads, 0, ctx->stream>>>(
                bucket_size, static_cast<uint32_t>(buckets), big, big_counters, big_items, big_buckets);
        }
        GZK_CUDA_TRY(ctx, cudaGetLastError());
        GZK_CUDA_TRY(ctx, cudaMemsetAsync(size_bins, 0, 2 * kSizeBins * sizeof(uint32_t), ctx->stream));
        {
            LaunchScope scope(ctx, "msm_order", 2);
            const unsigned blocks = static_cast<unsigned>((buckets + 1023) / 1024);
            msm_size_histogram_kernel<<<blocks, 1024, 0, ctx->stream>>>(bucket_size, static_cast<uint32_t>(buckets), big, size_bins);
            msm_order_kernel<<<blocks, 1024, 0, ctx->stream>>>(bucket_size, static_cast<uint32_t>(buckets), big, size_bins, size_bins + kSizeBins, order);
        }
        GZK_CUDA_TRY(ctx, cudaGetLastError());
        {
            LaunchScope scope(ctx, "msm_buckets");
            const uint32_t lanes = bucket_lanes(ctx, buckets, total_entries);
            const auto kernel = lanes == 1 ? msm_buckets_kernel<1> : lanes == 2 ? msm_buckets_kernel<2> : lanes == 4 ? msm_buckets_kernel<4> : msm_buckets_kernel<8>;
            kernel<<<static_cast<unsigned>((buckets * lanes + kThreads - 1) / kThreads), kThreads, 0, ctx->stream>>>(
                static_cast<const G1Affine*>(points->dptr), bucket_start, bucket_size, order, entries, static_cast<uint32_t>(buckets), big, bucket_points);
        }
        GZK_CUDA_TRY(ctx, cudaGetLastError());
        {
            // the counts stay on the device: grids that fill the chip, or the upper bound where that is less
            LaunchScope scope(ctx, "msm_big_buckets", 2);
            const uint64_t cap = static_cast<uint64_t>(ctx->sm_count) * 4;
            msm_big_slices_kernel<<<static_cast<unsigned>(max_items < cap ? max_items : cap), kThreads, 0, ctx->stream>>>(
                static_cast<const G1Affine*>(points->dptr), bucket_start, bucket_size, entries, big_counters, big_items, big_partial);
            msm_big_combine_kernel<<<static_cast<unsigned>(max_big < cap ? max_big : cap), kThreads, 0, ctx->stream>>>(
                big_counters, big_buckets, big_partial, bucket_points);
        }
        GZK_CUDA_TRY(ctx, cudaGetLastError());
        {
            LaunchScope scope(ctx, "msm_bits", 3);
            const uint32_t lines = split_rows + (1u << split_h);
            // a line by one warp while that leaves the chip short of warps, else by eight lanes (32 lanes add five
            // levels of a tree to each line: for one set of 2^16 buckets the shorter chain, for 26 sets the longer)
            if (static_cast<uint64_t>(lines) * bucket_sets <= static_cast<uint64_t>(ctx->sm_count) * 8)
                msm_rowcol_kernel<32><<<dim3((lines * 32 + kThreads - 1) / kThreads, bucket_sets), kThreads, 0, ctx->stream>>>(bucket_points, plan.half, split_h, split_rows, bit_partial);
            else
                msm_rowcol_kernel<8><<<dim3((lines * 8 + kThreads - 1) / kThreads, bucket_sets), kThreads, 0, ctx->stream>>>(bucket_points, plan.half, split_h, split_rows, bit_partial);
            msm_rowcol_bits_kernel<<<dim3(plan.c, bucket_sets), kThreads, 0, ctx->stream>>>(bit_partial, split_h, split_rows, bit_sums);
            msm_window_sums_kernel<<<bucket_sets, kThreads, 0, ctx->stream>>>(bit_sums, plan.c, window_sums);
        }
        GZK_CUDA_TRY(ctx, cudaGetLastError());
        // the shifts of the windows are one chain of c * w doublings: the host's part
        G1Xyzz sums[kMaxWindows];
        GZK_CUDA_TRY(ctx, cudaMemcpyAsync(sums, window_sums, bucket_sets * sizeof(G1Xyzz), cudaMemcpyDeviceToHost, ctx->stream));
        GZK_CUDA_TRY(ctx, cudaStreamSynchronize(ctx->stream));
        host_to_affine_bytes(host_horner(sums, bucket_sets, plan.c), out_host);
        return GZK_OK;
    }
}

namespace gzk
{
    int msm_run(gzk_ctx* ctx, const gzk_buf* scalars, const gzk_buf* points, uint64_t n, uint8_t out_host[96])
    {
        // Above 2^24 points the (point, window) list of one pass no longer fits the caches that the
        // counting sort and the bucket gathers live on (2^26 points in one pass run at a third of the rate
        // of 2^24): longer inputs are cut into ranges of 2^24 points and the range sums are added.
        constexpr uint64_t kRange = 1ULL << 24;
        if (n <= kRange) return msm_run_plan(ctx, scalars, points, n, make_plan(n), out_host);
        std::vector<uint8_t> partial;
        for (uint64_t first = 0; first < n; first += kRange)
        {
            const uint64_t count = n - first < kRange ? n - first : kRange;
            gzk_buf s_view = *scalars, p_view = *points;
            s_view.dptr = static_cast<char*>(scalars->dptr) + first * scalars->elem_bytes;
            s_view.count = count;
            s_view.owned = false;
            p_view.dptr = static_cast<char*>(points->dptr) + first * points->elem_bytes;
            p_view.count = count;
            p_view.owned = false;
            partial.resize(partial.size() + 96);
            const int rc = msm_run_plan(ctx, &s_view, &p_view, count, make_plan(count), partial.data() + partial.size() - 96);
            if (rc != GZK_OK) return rc;
        }
        if (gzk_g1_sum(partial.data(), partial.size() / 96, out_host) != GZK_OK) return fail(ctx, GZK_E_INVALID, "msm: range sums are not canonical points");
        return GZK_OK;
    }
}

using namespace gzk;

extern "C" unsigned gzk_msm_window_bits(size_t n)
{
    // Start from log2(n) - 3 (a few hundred entries per bucket, >= 2^15 buckets so that one bucket
    // set keeps every SM busy) and compare its neighbours by additions: n per window, 2 per bucket
    // for the reduction, and a surcharge when the top window is only a few bits wide (its handful
    // of buckets then take n / 2^bits points each and go through the slower cooperative path).
    unsigned log2n = 0;
    while ((static_cast<size_t>(1) << (log2n + 1)) <= n) ++log2n;
    int c0 = static_cast<int>(log2n) - 3;
    if (c0 < 16) c0 = 16;
    if (c0 > 23) c0 = 23;
    double best_cost = 0.0;
    unsigned best = static_cast<unsigned>(c0);
    for (int c = c0 - 1; c <= c0 + 1; ++c)
    {
        const uint32_t windows = windows_for(static_cast<uint32_t>(c));
        const uint32_t full = (255 + static_cast<uint32_t>(c) - 1) / static_cast<uint32_t>(c);
        const int top_bits = 255 - c * static_cast<int>(full - 1);
        // a window beyond ceil(255 / c) only receives the carries of the one below it: about n / 2 entries
        double cost = (static_cast<double>(full) + (windows > full ? 0.5 : 0.0)) * static_cast<double>(n) + 2.0 * static_cast<double>(1ULL << (c - 1));
        if (top_bits > 0 && top_bits < 12) cost += 1.5 * static_cast<double>(n);
        if (static_cast<double>(windows) * static_cast<double>(n) / static_cast<double>(1ULL << (c - 1)) > 768.0) cost += 4.0 * static_cast<double>(n);
        if (best_cost == 0.0 || cost < best_cost)
        {
            best_cost = cost;
            best = static_cast<unsigned>(c);
        }
    }
    return best;
}

extern "C" size_t gzk_msm_table_points(size_t n, unsigned window_bits)
{
    if (window_bits < 2 || window_bits > 24) return 0;
    return n * windows_for(window_bits);
}

extern "C" int gzk_msm_precompute(gzk_ctx* ctx, const gzk_buf* points, size_t n, unsigned window_bits, gzk_buf* table)
{
    if (ctx == nullptr) return GZK_E_INVALID;
    if (points == nullptr || table == nullptr || points->kind != GZK_KIND_G1 || table->kind != GZK_KIND_G1 || points->count < n)
        return fail(ctx, GZK_E_INVALID, "msm_precompute: points and table must be G1 buffers");
    if (window_bits < 8 || window_bits > 24) return fail(ctx, GZK_E_INVALID, "msm_precompute: window_bits must lie in [8, 24]");
    const uint32_t windows = windows_for(window_bits);
    if (table->count < n * windows || table->dptr == points->dptr) return fail(ctx, GZK_E_INVALID, "msm_precompute: table needs gzk_msm_table_points(n, window_bits) points of its own");
    if (n == 0) return GZK_OK;
    GZK_CUDA_TRY(ctx, cudaSetDevice(ctx->device));
    G1Affine* t = static_cast<G1Affine*>(table->dptr);
    GZK_CUDA_TRY(ctx, cudaMemcpyAsync(t, points->dptr, n * sizeof(G1Affine), cudaMemcpyDeviceToDevice, ctx->stream));
    for (uint32_t w = 1; w < windows; ++w)
    {
        LaunchScope scope(ctx, "msm_table_window");
        msm_table_window_kernel<<<static_cast<unsigned>((n + kThreads - 1) / kThreads), kThreads, 0, ctx->stream>>>(t + static_cast<size_t>(w - 1) * n,
                                                                                                          t + static_cast<size_t>(w) * n, n, window_bits);
    }
    GZK_CUDA_TRY(ctx, cudaGetLastError());
    return finish_call(ctx, "invalid input");
}

extern "C" int gzk_msm_precomputed(gzk_ctx* ctx, const gzk_buf* scalars, const gzk_buf* table, size_t n, unsigned window_bits, uint8_t out[96])
{
    if (ctx == nullptr) return GZK_E_INVALID;
    if (out == nullptr) return fail(ctx, GZK_E_INVALID, "msm_precomputed: null output");
    if (n == 0)
    {
        std::memset(out, 0, 96);
        return GZK_OK;
    }
    if (scalars == nullptr || table == nullptr) return fail(ctx, GZK_E_INVALID, "msm_precomputed: null argument");
    if (window_bits < 8 || window_bits > 24) return fail(ctx, GZK_E_INVALID, "msm_precomputed: window_bits must lie in [8, 24]");
    if ((scalars->kind != GZK_KIND_FR && scalars->kind != GZK_KIND_FR_MONT) || scalars->count < n)
        return fail(ctx, GZK_E_INVALID, "msm_precomputed: scalars must be an FR or FR_MONT buffer of n elements");
    const MsmPlan plan = make_shared_plan(window_bits);
    if (table->kind != GZK_KIND_G1 || table->count < n * plan.windows) return fail(ctx, GZK_E_INVALID, "msm_precomputed: table does not hold gzk_msm_table_points(n, window_bits) points");
    if (n * plan.windows >= (1ULL << 31)) return fail(ctx, GZK_E_INVALID, "msm_precomputed: at most 2^31 - 1 table points per call");
    GZK_CUDA_TRY(ctx, cudaSetDevice(ctx->device));
    return msm_run_plan(ctx, scalars, table, n, plan, out);
}

extern "C" int gzk_msm(gzk_ctx* ctx, const gzk_buf* scalars, const gzk_buf* points, size_t n, uint8_t out[96])
{
    if (ctx == nullptr) return GZK_E_INVALID;
    if (out == nullptr) return fail(ctx, GZK_E_INVALID, "msm: null output");
    if (n == 0)
    {
        std::memset(out, 0, 96);
        return GZK_OK;
    }
    if (scalars == nullptr || points == nullptr) return fail(ctx, GZK_E_INVALID, "msm: null argument");
    if ((scalars->kind != GZK_KIND_FR && scalars->kind != GZK_KIND_FR_MONT) || scalars->count < n)
        return fail(ctx, GZK_E_INVALID, "msm: scalars must be an FR or FR_MONT buffer of n elements");
    if (points->kind != GZK_KIND_G1 || points->count < n) return fail(ctx, GZK_E_INVALID, "msm: points must be a G1 buffer of n elements");
    // the counting sort addresses n * windows (point, window) entries with 32-bit offsets
    if (n * make_plan(n).windows >= (1ULL << 31)) return fail(ctx, GZK_E_INVALID, "msm: at most 2^31 - 1 (point, window) entries per call (about 2^26 points); split the point range and add the results with gzk_g1_sum");
    GZK_CUDA_TRY(ctx, cudaSetDevice(ctx->device));
    return msm_run(ctx, scalars, points, n, out);
}
