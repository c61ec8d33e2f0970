// wrs_sample.cu -- sampling kernels of the WRS hot path for sm_103a.
//
//   k_alias_sample  alias-table sampling      (reference: src/device/wrs/alias/sampling/shader.comp:68-111)
//   k_its_sample    inverse transform sampling by bisection over the CMF
//                                             (reference: src/device/wrs/its/sampling/shader.comp:80-177)
//
// Two generator modes:
//   RNG_REF      the shaders' own streams: Philox2x32-7 variant with counter (0, gid) and
//                key = seed for the alias method; wang_hash(seed + gid) for ITS.  Indices
//                are bit-exact with the shaders' arithmetic.
//   RNG_PHILOX   Random123 Philox4x32-10, key = (seed lo, seed hi), counter = (sample
//                index lo, hi, 0, 0).  Alias: ix = mulhi(x0, N); the bucket keeps ix when
//                p >= 1 or x1 < ceil(p * 2^32), else returns its alias (32-bit coin).
//                ITS: target T = (2*x0 + 1) * cmf[N-1] * 2^-33 in (0, total), formed
//                exactly in 64-bit integers and kept as its FP32 rounding plus the sign of
//                the rounding residual, so every probe "T > cmf[mid]" is decided exactly
//                with one FP32 compare; result = first index with cmf >= T.  Zero-weight
//                items can never be drawn.
#include "wrs_device.cuh"
#include "wrs_internal.cuh"

namespace wrs {

constexpr uint32_t RNG_REF = 0, RNG_PHILOX = 1;

// mix(x, y, a) evaluated as x*(1-a) + y*a, one rounding per operation
__device__ __forceinline__ float mix_rn(float x, float y, float a) {
    return __fadd_rn(__fmul_rn(x, __fsub_rn(1.0f, a)), __fmul_rn(y, a));
}

// The eighth of [0, 1) a float p or coin u lies in: 0 for p <= 0 and NaN, 7 for values of 1 and
// above (the product is exact, the conversion truncates and saturates).
__device__ __forceinline__ uint32_t coin_cell_f(float p) {
    return min(__float2uint_rz(__fmul_rn(p, 8.0f)), 7u);
}

// What a block says about a sample of bucket `self` whose coin lies in `cell`: the bucket itself,
// its alias, or nothing (need: the entry must be read).
struct BlockSays {
    uint32_t r;
    bool need;
};
__device__ __forceinline__ BlockSays block_says(const uint4& lo, const uint4& hi, uint32_t cell,
                                                uint32_t self) {
    const uint32_t b = self & 31u;
    const uint32_t code = ((lo.x >> b) & 1u) | ((lo.y >> b) & 1u) << 1 | ((lo.z >> b) & 1u) << 2;
    BlockSays s;
    s.r = self;
    s.need = cell == code;
    if (cell > code) {
        const uint32_t width = hi.x >> kAliasHeadBits;
        const uint32_t up = lo.w >> b;  // bit 0: this bucket is heavy; then the buckets above it
        if (up & 1u) {
            // the distance to the next heavy bucket (0: beyond the block)
            const uint32_t next = up & 0xfffffffeu;
            s.r = self + (31u - static_cast<uint32_t>(__clz(static_cast<int>(next & (0u - next)))));
            s.need = next == 0u || width == kAliasNone;
        } else {
            const uint32_t j = __popc(hi.y << (31u - b));  // switches up to this bucket
            uint32_t d;
            if (width == kAliasSteps) {
                // the sum of the first j nibbles, and j
                const uint64_t x = (static_cast<uint64_t>(hi.w) << 32 | hi.z) << (64u - 4u * j & 63u);
                const uint32_t x0 = static_cast<uint32_t>(x), x1 = static_cast<uint32_t>(x >> 32);
                d = __dp4a(x0 & 0x0f0f0f0fu, 0x01010101u, j);
                d = __dp4a(x0 >> 4 & 0x0f0f0f0fu, 0x01010101u, d);
                d = __dp4a(x1 & 0x0f0f0f0fu, 0x01010101u, d);
                d = __dp4a(x1 >> 4 & 0x0f0f0f0fu, 0x01010101u, d);
            } else {
                const uint64_t off =
                    (static_cast<uint64_t>(hi.w) << 32 | hi.z) >> ((j - 1u) * width & 63u);
                d = static_cast<uint32_t>(off) & (0xffffffffu >> (32u - width & 31u));
            }
            s.r = (hi.x & kAliasHeadMask) + (j ? d : 0u);
            s.need = width == kAliasNone;
        }
    }
    return s;
}

// Samples [(256 block + t) PT, +PT) of one distribution (thread t of the CTA).  BLOCKS: blocks are
// the table's alias blocks, consulted where `use` holds.
//
// By the table alone a sample is one random 8-byte read: from a table beyond L2 the device's rate of
// random HBM accesses bounds it (50-70 G/s, whatever the bytes), from one in L2 the L1's one
// wavefront per gathered sector (250 G/s).  Through the blocks (1 byte per bucket: 64 MB at n = 2^26,
// 22 % of whose reads miss L2 there) one 32-byte sector decides 86 % of uniform weights' samples.  The
// bounds are instruction issue (72 % active, ~150 instructions per 32 samples) and, at 2^26, the random
// accesses of block misses and entries together (16 bytes read from HBM a sample in fetches of 64: 40
// G/s): 2^28 samples, n = 2^26, uniform 2.76 -> 1.64 ms, log-normal(0, 2) 4.3 -> 1.73; 2 x 10^8
// samples, n = 5 x 10^7, Zipf 3.3 -> 1.10 ms (against one byte of p per bucket, which decided only the
// samples that their bucket keeps).
template <uint32_t RNG, bool COOP, bool BLOCKS, int PT = kAliasPerThread>
__device__ __forceinline__ void alias_block(const uint2* __restrict__ table,
                                            const AliasBlock* __restrict__ blocks, bool use,
                                            uint32_t n, uint64_t S, uint64_t seed,
                                            uint64_t offset, uint32_t coop,
                                            uint32_t* __restrict__ out, uint64_t block) {
    const uint64_t t = block * kSampleThreads + threadIdx.x;
    const uint64_t s0 = t * PT;
    if (s0 >= S) return;
    uint32_t r[PT], ixs[PT];
    uint32_t coin[PT];  // RNG_PHILOX: 32 bits; RNG_REF: the float coin's bits
    if constexpr (RNG == RNG_REF) {
        const uint32_t key = static_cast<uint32_t>(seed);
        const float fn = __uint2float_rn(n);
        float sx = 0.f, sy = 0.f;
        if constexpr (COOP) {
            // narrowSection (shader.comp:68-76): the subgroup's elected lane is the first
            // sample of its aligned group of 32; section = ix -/+ coop/2
            const uint32_t g0 = static_cast<uint32_t>(offset + (s0 & ~31ull));
            const uint2 u = philox2x32_7(0u, g0, key);
            const int ix = __float2int_rz(__fmul_rn(fn, unit_ref(u.x)));
            sx = __int2float_rn(ix - static_cast<int>(coop) / 2);
            sy = __int2float_rn(ix + static_cast<int>(coop) / 2);
        }
#pragma unroll
        for (int v = 0; v < PT; ++v) {
            const uint32_t g = static_cast<uint32_t>(offset + s0 + v);
            const uint2 u = philox2x32_7(0u, g, key);
            const float ux = unit_ref(u.x);
            coin[v] = __float_as_uint(unit_ref(u.y));
            const float f = COOP ? mix_rn(sx, sy, ux) : __fmul_rn(fn, ux);
            int ix = __float2int_rz(f);
            ix = ix < 0 ? 0 : ix;
            ix = ix > static_cast<int>(n - 1u) ? static_cast<int>(n - 1u) : ix;
            ixs[v] = static_cast<uint32_t>(ix);
        }
    } else {
        uint2 ks[10];
        philox4x32_10_keys(seed, ks);
#pragma unroll
        for (int v = 0; v < PT; ++v) {
            const uint64_t g = offset + s0 + v;
            const uint4 x = philox4x32_10(
                make_uint4(static_cast<uint32_t>(g), static_cast<uint32_t>(g >> 32), 0u, 0u), ks);
            ixs[v] = __umulhi(x.x, n);
            coin[v] = x.y;
        }
    }
    // whether the bucket keeps a sample, from its entry's p
    auto keeps = [&](uint32_t c, uint32_t pbits) {
        const float p = __uint_as_float(pbits);
        if constexpr (RNG == RNG_REF) return !(__uint_as_float(c) >= p);
        return p >= 1.0f || c < __float2uint_ru(__fmul_rn(p, 4294967296.0f));
    };
    bool blocked = false;
    if constexpr (BLOCKS) blocked = use;
    if (BLOCKS && blocked) {
        const uint64_t once = l2_policy_evict_first();  // table entries: keep the blocks in L2
        uint4 lo[PT], hi[PT];
        bool need[PT];
        uint2 ent[PT];
#pragma unroll
        for (int v = 0; v < PT; ++v)
            ld_block(reinterpret_cast<const uint32_t*>(blocks + (ixs[v] >> 5)), lo[v], hi[v]);
#pragma unroll
        for (int v = 0; v < PT; ++v) {
            const uint32_t cell =
                RNG == RNG_REF ? coin_cell_f(__uint_as_float(coin[v])) : coin[v] >> 29;
            const BlockSays s = block_says(lo[v], hi[v], cell, ixs[v]);
            r[v] = s.r;
            need[v] = s.need;
            if (s.need) ent[v] = ld_entry_policy(table + ixs[v], once);
        }
#pragma unroll
        for (int v = 0; v < PT; ++v)
            if (need[v]) r[v] = keeps(coin[v], ent[v].x) ? ixs[v] : ent[v].y;
    } else {
        uint2 ent[PT];
#pragma unroll
        for (int v = 0; v < PT; ++v) ent[v] = ld_entry(table + ixs[v]);
#pragma unroll
        for (int v = 0; v < PT; ++v)
            r[v] = keeps(coin[v], ent[v].x) ? ixs[v] : ent[v].y;
    }
    if (s0 + PT <= S && (reinterpret_cast<uintptr_t>(out) & (PT * 4u - 1u)) == 0) {
        if constexpr (PT == 4)
            __stcs(reinterpret_cast<uint4*>(out + s0), make_uint4(r[0], r[1], r[2], r[3]));
        else if constexpr (PT == 2)
            __stcs(reinterpret_cast<uint2*>(out + s0), make_uint2(r[0], r[1]));
        else
            __stcs(out + s0, r[0]);
    } else {
#pragma unroll
        for (int v = 0; v < PT; ++v)
            if (s0 + v < S) out[s0 + v] = r[v];
    }
}

template <uint32_t RNG, bool COOP, bool BLOCKS>
__global__ __launch_bounds__(kSampleThreads) void k_alias_sample(
    const uint2* __restrict__ table, const AliasBlock* __restrict__ blocks,
    const unsigned long long* __restrict__ reads, uint32_t n, uint64_t S, uint64_t seed,
    uint64_t offset, uint32_t coop, uint32_t* __restrict__ out) {
    pdl_wait();
    bool use = false;
    if constexpr (BLOCKS) use = __ldg(reads) <= static_cast<unsigned long long>(kBlockMaxReads) * n;
    alias_block<RNG, COOP, BLOCKS, BLOCKS ? kBlockPerThread : kAliasPerThread>(table, blocks, use, n, S, seed, offset, coop, out, blockIdx.x);
}

// All distributions of a batch in one launch: CTA b samples block b - sample0 of the
// distribution the map names, with that distribution's seed and counter = sample index,
// so each distribution draws exactly the samples a per-call wrs_sample would.
template <uint32_t RNG, bool COOP>
__global__ __launch_bounds__(kSampleThreads) void k_alias_sample_batch(BatchView bv,
                                                                       uint32_t coop) {
    pdl_wait();
    const uint32_t d = __ldg(bv.sample_map + blockIdx.x);
    const DistDesc* D = bv.dist + d;
    alias_block<RNG, COOP, false>(D->table, nullptr, false, D->n, D->s, D->seed, 0ull, coop,
                                  D->out, blockIdx.x - D->sample0);
}

// The alias blocks of table[0, n), one per thread, from its 32 entries (eight 32-byte loads, whole
// sectors) and the partition's heavy bits.  0.105-0.111 ms at n = 2^26 (5.6 TB/s; HBM and the ALU
// pipe about level).  One thread per block keeps the encoding serial and short, ~20 instructions per
// entry; a lane per bucket (ballots and shuffles) would issue three times as many, and staging the
// entries in shared memory for coalesced loads took 0.21 ms.  A block is encoded only where its aliases follow the rule that the
// sampler decodes; where one does not (overlapping subproblems, distances that do not fit, a NaN)
// the block keeps its codes and says so.  *reads receives 8 times the expected number of entry
// reads by one sample of every bucket.
__global__ __launch_bounds__(kBlockBuildThreads, 8) void k_alias_blocks(
    const uint2* __restrict__ table, const uint32_t* __restrict__ classes, uint32_t n,
    AliasBlock* __restrict__ blocks, unsigned long long* __restrict__ reads) {
    pdl_wait();
    __shared__ uint32_t s_sum[kBlockBuildThreads / 32];
    const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31u;
    const uint64_t base64 =
        (static_cast<uint64_t>(blockIdx.x) * kBlockBuildThreads + threadIdx.x) * 32u;
    uint32_t sum = 0;
    if (base64 < n) {
        const uint32_t base = static_cast<uint32_t>(base64);
        const uint32_t live = n - base >= 32u ? 0xffffffffu : (1u << (n - base)) - 1u;
        const uint2* row = table + base;
        const uint32_t cls = __ldg(classes + (base >> 5)) & live;
        const uint32_t lights = ~cls & live;
        const uint32_t head = lights ? __ldg(&row[__ffs(lights) - 1].y) : 0u;
        uint32_t p0 = 0, p1 = 0, p2 = 0, sw = 0, odd = 0;
        float nan = 0.0f;  // NaN once a p is (or is infinite)
        uint32_t alias = head, heavy_alias = cls ? base + __ffs(cls) - 1u : 0u;
        uint32_t step_max = 0, step_lo = 0, step_hi = 0;
#pragma unroll
        for (int q = 0; q < 8; ++q) {
            uint4 lo = make_uint4(0u, 0u, 0u, 0u), hi = lo;
            if (live == 0xffffffffu) {
                ld_block(reinterpret_cast<const uint32_t*>(row + 4 * q), lo, hi);
            } else {
                uint2 e[4];
#pragma unroll
                for (int c = 0; c < 4; ++c)
                    e[c] = live >> (4 * q + c) & 1u ? __ldg(row + 4 * q + c) : make_uint2(0u, 0u);
                lo = make_uint4(e[0].x, e[0].y, e[1].x, e[1].y);
                hi = make_uint4(e[2].x, e[2].y, e[3].x, e[3].y);
            }
            const uint32_t px[4] = {lo.x, lo.z, hi.x, hi.z}, al[4] = {lo.y, lo.w, hi.y, hi.w};
#pragma unroll
            for (int c = 0; c < 4; ++c) {
                const int i = 4 * q + c;
                // p in [0, 1): floor(2 p), floor(4 p) and floor(8 p) in the low mantissa bits of
                // 2^23 + k p rounded down (on the FMA pipe; the ALU pipe is the busier one)
                const float p = __uint_as_float(px[c]);
                const float q = fminf(__saturatef(p), 0x1.fffffep-1f);
                p0 = __funnelshift_r(p0, __float_as_uint(__fmaf_rz(q, 8.0f, 8388608.0f)), 1);
                p1 = __funnelshift_r(p1, __float_as_uint(__fmaf_rz(q, 4.0f, 8388608.0f)), 1);
                p2 = __funnelshift_r(p2, __float_as_uint(__fmaf_rz(q, 2.0f, 8388608.0f)), 1);
                nan = __fmaf_rn(p, 0.0f, nan);
                const bool heavy = (cls & 1u << i) != 0u;
                // the heavy bucket before does not alias this one
                if (heavy && heavy_alias != base + i) odd |= 1u << i;
                heavy_alias = heavy ? al[c] : heavy_alias;
                // a light bucket with another alias than the light one before
                const uint32_t step = al[c] - alias - 1u;  // (wraps where the aliases do not rise)
                if (!heavy && step != 0xffffffffu) {
                    sw |= 1u << i;
                    step_lo = __funnelshift_r(step_lo, step_hi, 4);
                    step_hi = __funnelshift_r(step_hi, step, 4);
                    step_max = max(step_max, step);
                }
                alias = heavy ? alias : al[c];
            }
        }
        const bool whole = live == 0xffffffffu;
        sw &= live;
        const uint32_t m = __popc(sw);
        uint64_t off = 0;
        uint32_t code = kAliasNone;
        if (nan == 0.0f && odd == 0u && head <= kAliasHeadMask) {
            if (whole && m <= 16u && step_max <= 15u) {
                code = kAliasSteps;
                off = m ? (static_cast<uint64_t>(step_hi) << 32 | step_lo) >> (64u - 4u * m) : 0u;
            } else {
                const uint32_t width = min(64u / max(m, 1u), 31u);  // bits per distance
                uint32_t far = 0, at = 0;
                for (uint32_t rest = sw; rest; rest &= rest - 1u, at += width) {
                    const uint32_t d = __ldg(&row[__ffs(rest) - 1].y) - head;
                    off |= static_cast<uint64_t>(d) << at;
                    far |= d;
                }
                if (width > kAliasSteps && far >> width == 0u) code = width;
            }
        }
        uint4* dst = reinterpret_cast<uint4*>(blocks + (base >> 5));
        dst[0] = make_uint4(p0, p1, p2, cls);
        dst[1] = make_uint4((head & kAliasHeadMask) | code << kAliasHeadBits, sw,
                            static_cast<uint32_t>(off), static_cast<uint32_t>(off >> 32));
        // entry reads, in eighths of a sample per bucket: coins in the bucket's own cell, or all
        // above it
        sum = __popc(live);
        if (code == kAliasNone)
            sum = 8u * sum - __popc(p0 & live) - 2u * __popc(p1 & live) - 4u * __popc(p2 & live);
    }
    sum = __reduce_add_sync(0xffffffffu, sum);
    if (lane == 0) s_sum[warp] = sum;
    __syncthreads();
    if (threadIdx.x == 0) {
        uint32_t tot = 0;
        for (int w = 0; w < kBlockBuildThreads / 32; ++w) tot += s_sum[w];
        atomicAdd(reads, static_cast<unsigned long long>(tot));
    }
}

// its/sampling/shader.comp:80-94
__device__ __forceinline__ float search_range_u(const float* __restrict__ cmf, uint32_t x,
                                                uint32_t y, float u) {
    const float lo = x > 0 ? __ldg(cmf + x - 1) : 0.0f;
    const float hi = __ldg(cmf + y);
    return __fadd_rn(lo, __fmul_rn(__fsub_rn(hi, lo), u));
}

// its/sampling/shader.comp:131-140: lower bound with the shader's probe sequence
__device__ __forceinline__ uint32_t bisect(const float* __restrict__ cmf, uint32_t x, uint32_t y,
                                           float u) {
    while (x < y) {
        const uint32_t mid = x + ((y - x) >> 1);
        if (u > __ldg(cmf + mid))
            x = mid + 1;
        else
            y = mid;
    }
    return x;
}

// T = (2x + 1) * total * 2^-33 as (t_hi = T rounded to nearest FP32, t_sgn = sign(T - t_hi)).
// total = Mt * 2^Et with a 24-bit integer Mt; P = (2x + 1) * Mt < 2^57 is exact in 64 bits.
__device__ __forceinline__ void exact_target(uint32_t x, float total, float& t_hi, int& t_sgn) {
    const uint32_t tb = __float_as_uint(total);
    const int e = static_cast<int>((tb >> 23) & 0xffu);
    const uint64_t mt = e ? ((tb & 0x7fffffu) | 0x800000u) : (tb & 0x7fffffu);
    const int et = (e ? e : 1) - 150;
    const uint64_t P = (2ull * x + 1ull) * mt;
    if (P == 0) {
        t_hi = 0.0f;
        t_sgn = 0;
        return;
    }
    const int bits = 64 - __clzll(static_cast<long long>(P));
    int sh = bits > 24 ? bits - 24 : 0;
    uint64_t mant = P >> sh;
    int sgn = 0;
    if (sh > 0) {
        const uint64_t rem = P & ((1ull << sh) - 1ull), half = 1ull << (sh - 1);
        if (rem > half || (rem == half && (mant & 1ull))) {
            ++mant;
            sgn = -1;
        } else {
            sgn = rem ? 1 : 0;
        }
        if (mant == (1ull << 24)) {
            mant >>= 1;
            ++sh;
        }
    }
    t_hi = ldexpf(static_cast<float>(mant), et - 33 + sh);
    t_sgn = sgn;
}

// first index in [0, last] with cmf >= T, bisecting like its/sampling/shader.comp:131-140
__device__ __forceinline__ uint32_t bisect_exact(const float* __restrict__ cmf, uint32_t last,
                                                 float t_hi, int t_sgn) {
    uint32_t x = 0, y = last;
    while (x < y) {
        const uint32_t mid = x + ((y - x) >> 1);
        const float c = __ldg(cmf + mid);
        if (t_hi > c || (t_hi == c && t_sgn > 0))
            x = mid + 1;
        else
            y = mid;
    }
    return x;
}

// COOP: 0 = none, 1 = binary narrowing, 2 = p-array narrowing.  One sample per thread so a
// warp is the shader's subgroup of 32 consecutive samples; every lane of the warp takes
// part in the narrowing (also lanes past S in the last warp, which then store nothing).
template <uint32_t RNG, int COOP>
__global__ __launch_bounds__(kSampleThreads) void k_its_sample(const float* __restrict__ cmf,
                                                               uint32_t n, uint64_t S,
                                                               uint64_t seed, uint64_t offset,
                                                               uint32_t coop,
                                                               uint32_t* __restrict__ out) {
    pdl_wait();
    const uint64_t s = static_cast<uint64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
    if constexpr (COOP == 0) {
        if (s >= S) return;
    } else {
        if ((s & ~31ull) >= S) return;  // whole warps only
    }
    uint32_t res;
    if constexpr (RNG == RNG_REF) {
        const uint32_t seed32 = static_cast<uint32_t>(seed);
        const uint32_t g = static_cast<uint32_t>(offset + s);
        uint32_t x = 0, y = n - 1u;
        if constexpr (COOP != 0) {
            const int lane = threadIdx.x & 31;
            const uint32_t g0 = __shfl_sync(0xffffffffu, g, 0);
            const float u1 =
                __shfl_sync(0xffffffffu, search_range_u(cmf, 0, n - 1u, unit_ref(wang_hash(seed32 + g0))), 0);
            if constexpr (COOP == 2) {
                uint32_t range = y - x + 1u;
                while (range > coop) {
                    const uint32_t base = range / 32u;
                    const uint32_t start = x + lane * base;
                    uint32_t end = start + base - 1u;
                    end = end > y ? y : end;
                    const unsigned b = __ballot_sync(0xffffffffu, u1 < __ldg(cmf + end));
                    if (b) {
                        const int id = __ffs(b) - 1;
                        x = __shfl_sync(0xffffffffu, start, id);
                        y = __shfl_sync(0xffffffffu, end, id);
                    } else {
                        // u1 beyond every partition end (the shader's ballot is empty there):
                        // keep the remainder, at least the last item
                        x = min(x + 32u * base, y);
                    }
                    range = y - x + 1u;
                }
            } else {
                while (y - x + 1u > coop) {
                    const uint32_t mid = x + ((y - x) >> 1);
                    if (u1 > __ldg(cmf + mid))
                        x = mid + 1;
                    else
                        y = mid;
                }
            }
        }
        const float u2 = search_range_u(cmf, x, y, unit_ref(wang_hash((seed32 ^ 0xA9EC5C80u) + g)));
        res = bisect(cmf, x, y, u2);
    } else {
        uint2 ks[10];
        philox4x32_10_keys(seed, ks);
        const uint64_t g = offset + s;
        const uint4 r = philox4x32_10(
            make_uint4(static_cast<uint32_t>(g), static_cast<uint32_t>(g >> 32), 0u, 0u), ks);
        float t_hi;
        int t_sgn;
        exact_target(r.x, __ldg(cmf + n - 1u), t_hi, t_sgn);
        res = bisect_exact(cmf, n - 1u, t_hi, t_sgn);
    }
    if (s < S) __stcs(out + s, res);
}

// ---- ITS without cooperative narrowing: the bisection's probe tree, top cached ----------
//
// Every non-cooperative search starts with x = 0, y = N - 1 and probes mid = x + (y - x) / 2,
// so its first probes walk one implicit binary tree: node k (root 1; children 2k for
// "T <= cmf[mid]" and 2k + 1 for "T > cmf[mid]") holds the range left by the branch
// decisions spelled by the bits of k below its leading one.  Each CTA copies the probe
// values of the top kItsTreeLevels levels into shared memory once, then runs the searches
// -- unchanged probe sequence, so results are bit-identical to the plain bisection -- with
// kItsPerThread searches interleaved per thread to keep several loads in flight.
constexpr int kItsTreeLevels = 12;
constexpr int kItsTreeNodes = 1 << kItsTreeLevels;  // nodes 1 .. 4095 (index 0 unused)
constexpr int kItsPerThread = 4;
constexpr int kItsGroup = kSampleThreads * kItsPerThread;
constexpr int kItsMaxBlocks = 152 * 16;

__device__ __forceinline__ void tree_range(uint32_t k, uint32_t last, uint32_t& x, uint32_t& y) {
    x = 0;
    y = last;
    const int d = 31 - __clz(k);
    for (int b = d - 1; b >= 0; --b) {
        if (x >= y) return;
        const uint32_t mid = x + ((y - x) >> 1);
        if ((k >> b) & 1u)
            x = mid + 1;
        else
            y = mid;
    }
}

static_assert(kItsTreeLevels == static_cast<int>(kTreeTop), "shared levels above the blocks");

// One thread per stored block (TreeBlock): the range of its root node, then the ranges of the
// root's 6 descendants and the probe values of the 7 nodes (0 for a node whose range is one
// index: no search reaches it with a probe).  Slot 7 holds the root's range [x, x + len - 1]
// as x | (len - floor(n / 2^level)) << 31: the ranges of one tree level are floor(n / 2^level)
// or one more long (the left half of a range takes the odd index), and x < 2^31.
__global__ __launch_bounds__(kSampleThreads) void k_its_tree(const float* __restrict__ cmf,
                                                             uint32_t n, uint32_t L,
                                                             TreeBlock* __restrict__ blocks) {
    pdl_wait();
    static_assert(its_tree_blocks(kTopBlockLevels) == kTopBlocks, "top block count");
    const size_t gb = static_cast<size_t>(blockIdx.x) * blockDim.x + threadIdx.x;
    if (gb >= its_tree_blocks(L)) return;
    uint32_t level = 0;
    size_t off = 0;
    while (gb >= off + (size_t(1) << level)) {
        off += size_t(1) << level;
        level += kTreeBlockLevels;
    }
    uint32_t xs[8], ys[8];
    tree_range((1u << level) + static_cast<uint32_t>(gb - off), n - 1u, xs[1], ys[1]);
    float v[8];
#pragma unroll
    for (int j = 1; j < 8; ++j) {
        const bool live = xs[j] < ys[j];
        const uint32_t mid = xs[j] + ((ys[j] - xs[j]) >> 1);
        v[j - 1] = live ? __ldg(cmf + mid) : 0.0f;
        if (j < 4) {
            // children: a finished range leaves finished ones
            xs[2 * j] = xs[j];
            ys[2 * j] = live ? mid : xs[j];
            xs[2 * j + 1] = live ? mid + 1 : xs[j];
            ys[2 * j + 1] = live ? ys[j] : xs[j];
        }
    }
    v[7] = __uint_as_float(xs[1] | ((ys[1] - xs[1] + 1u - (n >> level)) << 31));
    float4* dst = reinterpret_cast<float4*>(blocks + gb);
    dst[0] = make_float4(v[0], v[1], v[2], v[3]);
    dst[1] = make_float4(v[4], v[5], v[6], v[7]);
}

// With stored blocks (B > 0, so n > 2^16) no range ends above the tail: the ranges of tree
// level l hold at least floor(n / 2^l) >= 4 indices for every l below the last block level's
// bottom.  The shared and all but the last block levels then only follow the node (its probe
// value is the tree's); the last block's slot 7 gives the range of its root, and the searches
// track their ranges from there.  A decision is one comparison: "T > c" (the exact target's
// tie rule folded into the FP32 target: T_hi + a positive remainder is > c exactly when the
// next float above T_hi is > c).
template <uint32_t RNG>
__global__ __launch_bounds__(kSampleThreads) void k_its_sample_tree(const float* __restrict__ cmf,
                                                                    uint32_t n, uint64_t S,
                                                                    uint64_t seed, uint64_t offset,
                                                                    uint32_t* __restrict__ out,
                                                                    const TreeBlock* __restrict__ blocks,
                                                                    uint32_t B) {
    pdl_wait();
    __shared__ float s_tree[kItsTreeNodes];
    const uint32_t last = n - 1u;
    for (uint32_t k = threadIdx.x + 1; k < kItsTreeNodes; k += blockDim.x) {
        uint32_t x, y;
        tree_range(k, last, x, y);
        s_tree[k] = x < y ? __ldg(cmf + x + ((y - x) >> 1)) : 0.0f;
    }
    __syncthreads();
    const float total = __ldg(cmf + last);
    for (uint64_t grp = blockIdx.x; grp * kItsGroup < S; grp += gridDim.x) {
        const uint64_t s0 = grp * kItsGroup + threadIdx.x;
        float t[kItsPerThread];  // a search goes right at probe c exactly when t > c
        uint32_t x[kItsPerThread], y[kItsPerThread], node[kItsPerThread];
        if constexpr (RNG == RNG_REF) {
            const uint32_t seed32 = static_cast<uint32_t>(seed);
#pragma unroll
            for (int v = 0; v < kItsPerThread; ++v) {
                const uint32_t g = static_cast<uint32_t>(offset + s0 + v * kSampleThreads);
                t[v] = search_range_u(cmf, 0, last, unit_ref(wang_hash((seed32 ^ 0xA9EC5C80u) + g)));
            }
        } else {
            uint2 ks[10];
            philox4x32_10_keys(seed, ks);
#pragma unroll
            for (int v = 0; v < kItsPerThread; ++v) {
                const uint64_t g = offset + s0 + v * kSampleThreads;
                const uint4 r = philox4x32_10(
                    make_uint4(static_cast<uint32_t>(g), static_cast<uint32_t>(g >> 32), 0u, 0u), ks);
                float t_hi;
                int t_sgn;
                exact_target(r.x, total, t_hi, t_sgn);
                // t_hi >= 0: the next float above is one bit pattern up (+inf above the largest)
                t[v] = t_sgn > 0 ? __uint_as_float(__float_as_uint(t_hi) + 1u) : t_hi;
            }
        }
        if (B > 0) {
#pragma unroll
            for (int v = 0; v < kItsPerThread; ++v) node[v] = 1;
#pragma unroll
            for (int l = 0; l < kItsTreeLevels; ++l)
#pragma unroll
                for (int v = 0; v < kItsPerThread; ++v)
                    node[v] = 2 * node[v] + (t[v] > s_tree[node[v]] ? 1u : 0u);
            const TreeBlock* level_blocks = blocks;
            uint32_t level = kTreeTop;
#pragma unroll 1
            for (uint32_t bl = 0; bl < B; ++bl, level += kTreeBlockLevels) {
                const uint32_t first = 1u << level;  // the level's first node
                uint4 lo[kItsPerThread], hi[kItsPerThread];
#pragma unroll
                for (int v = 0; v < kItsPerThread; ++v)
                    ld_u32x8(reinterpret_cast<const uint32_t*>(level_blocks + (node[v] - first)),
                             lo[v], hi[v]);
                level_blocks += first;
                if (bl + 1 < B) {
#pragma unroll
                    for (int v = 0; v < kItsPerThread; ++v) {
                        const uint32_t r0 = t[v] > __uint_as_float(lo[v].x) ? 1u : 0u;
                        const uint32_t r1 =
                            t[v] > __uint_as_float(r0 ? lo[v].z : lo[v].y) ? 1u : 0u;
                        const uint32_t c2 = r0 ? (r1 ? hi[v].z : hi[v].y) : (r1 ? hi[v].x : lo[v].w);
                        const uint32_t r2 = t[v] > __uint_as_float(c2) ? 1u : 0u;
                        node[v] = 8 * node[v] + 4 * r0 + 2 * r1 + r2;
                    }
                } else {
                    const uint32_t floor_len = n >> level;
#pragma unroll
                    for (int v = 0; v < kItsPerThread; ++v) {
                        x[v] = hi[v].w & 0x7fffffffu;
                        y[v] = x[v] + floor_len + (hi[v].w >> 31) - 1u;
                        uint32_t mid = x[v] + ((y[v] - x[v]) >> 1);
                        const uint32_t r0 = t[v] > __uint_as_float(lo[v].x) ? 1u : 0u;
                        x[v] = r0 ? mid + 1 : x[v];
                        y[v] = r0 ? y[v] : mid;
                        mid = x[v] + ((y[v] - x[v]) >> 1);
                        const uint32_t r1 =
                            t[v] > __uint_as_float(r0 ? lo[v].z : lo[v].y) ? 1u : 0u;
                        x[v] = r1 ? mid + 1 : x[v];
                        y[v] = r1 ? y[v] : mid;
                        mid = x[v] + ((y[v] - x[v]) >> 1);
                        const uint32_t c2 = r0 ? (r1 ? hi[v].z : hi[v].y) : (r1 ? hi[v].x : lo[v].w);
                        const uint32_t r2 = t[v] > __uint_as_float(c2) ? 1u : 0u;
                        x[v] = r2 ? mid + 1 : x[v];
                        y[v] = r2 ? y[v] : mid;
                        // the tail reads stay inside the CMF whatever the block holds
                        y[v] = min(y[v], last);
                        x[v] = min(x[v], y[v]);
                    }
                }
            }
#pragma unroll
            for (int v = 0; v < kItsPerThread; ++v)
                if (s0 + v * kSampleThreads >= S) y[v] = x[v];  // past the end: no tail loads
        } else {
            // the shared levels with ranges (short CMFs end inside them)
#pragma unroll
            for (int v = 0; v < kItsPerThread; ++v) {
                x[v] = 0;
                y[v] = s0 + v * kSampleThreads < S ? last : 0u;
                node[v] = 1;
            }
#pragma unroll 1
            for (int l = 0; l < kItsTreeLevels; ++l) {
#pragma unroll
                for (int v = 0; v < kItsPerThread; ++v) {
                    if (x[v] < y[v]) {
                        const uint32_t mid = x[v] + ((y[v] - x[v]) >> 1);
                        if (t[v] > s_tree[node[v]]) {
                            x[v] = mid + 1;
                            node[v] = 2 * node[v] + 1;
                        } else {
                            y[v] = mid;
                            node[v] = 2 * node[v];
                        }
                    }
                }
            }
        }
        // remaining levels from global memory, the searches' loads issued together
        for (;;) {
            float c[kItsPerThread];
            bool any = false;
#pragma unroll
            for (int v = 0; v < kItsPerThread; ++v) {
                any = any || x[v] < y[v];
                c[v] = x[v] < y[v] ? __ldg(cmf + x[v] + ((y[v] - x[v]) >> 1)) : 0.0f;
            }
            if (!any) break;
#pragma unroll
            for (int v = 0; v < kItsPerThread; ++v) {
                if (x[v] < y[v]) {
                    const uint32_t mid = x[v] + ((y[v] - x[v]) >> 1);
                    if (t[v] > c[v])
                        x[v] = mid + 1;
                    else
                        y[v] = mid;
                }
            }
        }
#pragma unroll
        for (int v = 0; v < kItsPerThread; ++v)
            if (s0 + v * kSampleThreads < S) __stcs(out + s0 + v * kSampleThreads, x[v]);
    }
}

// ---- ITS through cells ---------------------------------------------------------------------
//
// On a non-decreasing CMF every lower-bound search returns the same index, so the search can
// start anywhere that brackets the answer.  The compensated scan's CMF is non-decreasing by
// construction: its grid is below (ItsGrid).  The FP32 scan's CMF nearly is: its cells (ItsCell)
// are read where a target cannot meet a decrease (below), as follows.
// The CMF's range is cut into G = ceil(N / entry) cells of equal mass, the
// Cutpoint guiding table's: cell k starts at x_k = lower bound of c_k = fl(fl(total / G) * k),
// and a target T with c_k < T <= c_{k+1} has its lower bound in [x_k, y_k], y_k = x_{k+1}
// (N - 1 for the last cell).  Cell k is stored as one 32-byte block (ItsCell): x_k, y_k and,
// for the range cut into kCellParts parts of d = ceil((y - x + 1) / kCellParts) indices, the
// CMF at the last index of each part (min(x + (j + 1) d - 1, y)).  A sample finds its cell (an
// FP32 estimate moved by exact comparisons against c_k), reads the block with one 32-byte
// load -- one random sector, what an alias-table entry costs (a random 64-byte read costs
// about twice that on GB300) -- and the first part whose last value is >= T holds the lower
// bound: with d = 1 (cells of at most kCellParts candidates) that is the answer, otherwise a
// bisection of the part's d indices of the CMF finds it.  A target above the block's last
// value (a cell estimate that did not settle) falls back to the bisection of [0, N - 1].
// Results equal the bisection's (k_its_sample_tree's).

// Starts x_k = lower bound of c_k = fl(step * k) (clamped to N - 1) of the equal-mass cells of
// a non-decreasing CMF, in two passes, the first bracketing the second (c_k is non-decreasing in k,
// so x_k is too).  k_cell_groups bisects the whole CMF for the first start of every group of 32
// cells; then one warp per group finds its 32 starts in the group's bracket [x_{32g},
// x_{32(g+1)}]: where that holds at most 128 values, the lanes load them with one coalesced
// pass and each start is the bracket's start plus the number of values below its threshold,
// found by a bisection over the values held in the warp's registers (shuffles, no dependent
// loads); wider brackets are bisected in memory.
//
// GRID: the thresholds of the compensated ITS grid, c_k = 128 k 2^-s, exact for k <= 2^24.
// 2^s for a CMF of the given total and at most G cells: floor(total * 2^s) < 128 G (and within a
// factor of two of it, but for totals below 2^-96, whose power is capped)
__device__ __forceinline__ int its_shift(float total, uint32_t G) {
    const uint32_t e = __float_as_uint(total) >> 23;
    if (e == 0u) return 127;           // zero or denormal: F < 2^(127 - 126) steps
    // infinite (the weights' sum exceeds FP32's range): finite values are below 4 steps, all in cell 0,
    // the others start at the first infinite one (NaN or negative: results are meaningless)
    if (e >= 255u) return -126;
    const int E = 31 - __clz(static_cast<int>(G));
    // total = m 2^(e - 127), 1 <= m < 2: total * 2^s / 128 = m 2^E or half of it
    const float m = __uint_as_float((__float_as_uint(total) & 0x7fffffu) | 0x3f800000u);
    const bool half = __fmul_rn(m, __uint_as_float(static_cast<uint32_t>(E + 127) << 23)) >=
                      __uint2float_rn(G);
    return min(E - (static_cast<int>(e) - 127) - (half ? 1 : 0) + 7, 127);
}
__device__ __forceinline__ float pow2f(int e) {
    return __uint_as_float(static_cast<uint32_t>(e + 127) << 23);
}

template <bool GRID>
__device__ __forceinline__ float cell_step(const float* __restrict__ cmf, uint32_t n, uint32_t G) {
    const float total = __ldg(cmf + n - 1u);
    if constexpr (GRID) return pow2f(min(7 - its_shift(total, G), 128));  // (2^128: infinite)
    return __fdiv_rn(total, __uint2float_rn(G));
}
// threshold c_k of cell k
__device__ __forceinline__ float cell_at(float step, uint32_t k) {
    return k ? __fmul_rn(step, __uint2float_rn(k)) : 0.0f;
}

//
// The first pass is one thread per group that waits for each probe, so it reads the seven midpoints
// that the next three levels may probe together (bisect_ahead: bisect's probes and result on any CMF).
// n = 2^22, 4096 groups (the Cutpoint configuration's pass): a pass over every 1024th start and one
// inside its brackets, a probe at a time, 185.9 us; both three levels at a time 182.1 (two: 182.2,
// four: 184.1); one pass over the whole CMF 177.8.  ITS grid of 2^24 weights 535.6, 530, 523.4; of 2^27
// (512 K groups) a build 920 with the pass between, 913 without: it is gone.
__device__ __forceinline__ uint32_t bisect_ahead(const float* __restrict__ cmf, uint32_t x,
                                                 uint32_t y, float u) {
    constexpr int kLevels = 3, kNodes = (1 << kLevels) - 1;  // node k's children: 2k + 1 (down), 2k + 2 (up)
    while (x < y) {
        uint32_t lo[kNodes], hi[kNodes];
        float v[kNodes];
        lo[0] = x;
        hi[0] = y;
#pragma unroll
        for (int k = 0; k < kNodes; ++k) {
            const uint32_t mid = lo[k] + ((hi[k] - lo[k]) >> 1);
            const bool live = lo[k] < hi[k];
            v[k] = live ? __ldg(cmf + mid) : 0.f;
            if (2 * k + 2 < kNodes) {  // (a dead node's children: dead)
                lo[2 * k + 1] = lo[k];
                hi[2 * k + 1] = mid;
                lo[2 * k + 2] = live ? mid + 1u : lo[k];
                hi[2 * k + 2] = hi[k];
            }
        }
        int at = 0;  // the node's place in its level
#pragma unroll
        for (int level = 0; level < kLevels; ++level) {
            if (x >= y) break;
            float c = v[(1 << level) - 1];
#pragma unroll
            for (int q = 1; q < 1 << level; ++q) c = at == q ? v[(1 << level) - 1 + q] : c;
            const uint32_t mid = x + ((y - x) >> 1);
            const bool up = u > c;
            if (up)
                x = mid + 1u;
            else
                y = mid;
            at = 2 * at + (up ? 1 : 0);
        }
    }
    return x;
}
// group[g] = x_{32 g} (N - 1 past the last cell), g <= ceil(G / 32)
template <bool GRID>
__device__ __forceinline__ uint32_t group_start(const float* __restrict__ cmf, uint32_t n, uint32_t G,
                                                uint32_t g) {
    const uint64_t k = static_cast<uint64_t>(g) * 32u;
    return k < G ? bisect_ahead(cmf, 0, n - 1u,
                                cell_at(cell_step<GRID>(cmf, n, G), static_cast<uint32_t>(k)))
                 : n - 1u;
}
template <bool GRID>
__global__ __launch_bounds__(kSampleThreads) void k_cell_groups(const float* __restrict__ cmf,
                                                                uint32_t n, uint32_t G,
                                                                uint32_t* __restrict__ group) {
    pdl_wait();
    const uint32_t g = blockIdx.x * blockDim.x + threadIdx.x;
    if (g < group_entries(G)) group[g] = group_start<GRID>(cmf, n, G, g);
}

// The start of cell k = 32 g + lane (all lanes of the warp call it; k >= G returns N - 1), and
// the end of the group's bracket in hi.  OWN: without the first pass, the bracket's ends by the first
// two lanes' bisections.
template <bool GRID, bool OWN>
__device__ __forceinline__ uint32_t cell_start_warp(const float* __restrict__ cmf, uint32_t n,
                                                    uint32_t G, const uint32_t* __restrict__ group,
                                                    uint32_t g, uint32_t& hi) {
    const uint32_t lane = threadIdx.x & 31u;
    uint32_t lo;
    if constexpr (OWN) {
        uint32_t end = 0;
        if (lane < 2u) end = group_start<GRID>(cmf, n, G, g + lane);
        lo = __shfl_sync(0xffffffffu, end, 0);
        hi = __shfl_sync(0xffffffffu, end, 1);
    } else {
        lo = __ldg(group + g);
        hi = __ldg(group + g + 1u);
    }
    const uint32_t k = g * 32u + lane;
    const float t = k < G ? cell_at(cell_step<GRID>(cmf, n, G), k) : __int_as_float(0x7f800000);
    uint32_t x;
    if (hi >= lo && hi - lo < 128u) {
        // values lo .. lo + 127, 4 consecutive per lane (past hi or N: +inf, never below t)
        float v[4];
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            const uint32_t pos = lo + 4u * lane + q;
            v[q] = pos <= hi && pos < n ? __ldg(cmf + pos) : __int_as_float(0x7f800000);
        }
        // the values are non-decreasing across the lanes: find the first lane whose last
        // value is >= t (a bisection over the lanes' maxima, fixed trip count so that every
        // lane takes part in every shuffle), then count inside its 4 values
        uint32_t a = 0, b = 32;
#pragma unroll
        for (int it = 0; it < 6; ++it) {
            const uint32_t mid = (a + b) >> 1;
            const float m = __shfl_sync(0xffffffffu, v[3], min(mid, 31u));
            if (a < b) {
                if (m < t)
                    a = mid + 1u;
                else
                    b = mid;
            }
        }
        const uint32_t c = min(a, 31u);
        uint32_t in = 0;
#pragma unroll
        for (int q = 0; q < 4; ++q) in += __shfl_sync(0xffffffffu, v[q], c) < t ? 1u : 0u;
        const uint32_t cnt = a < 32u ? 4u * a + in : 128u;
        x = min(lo + cnt, hi);
    } else {
        x = k < G ? bisect(cmf, lo, hi > lo ? hi : lo, t) : n - 1u;
    }
    return k < G ? x : n - 1u;
}

// bit 31 of a cell's y: an FP32 CMF's cell the search cannot serve (the search bisects it)
constexpr uint32_t kCellUnsafe = 0x80000000u;

__device__ __forceinline__ uint32_t cell_part(uint32_t x, uint32_t y) {
    return (y - x + kCellParts) / kCellParts;  // ceil((y - x + 1) / kCellParts)
}

// the FP32 CMF need not be monotone: a cell whose start x > 0 does not have cmf[x - 1] < c_k is
// marked for the bisection as it is written
template <bool OWN>
__global__ __launch_bounds__(kSampleThreads) void k_its_cells(const float* __restrict__ cmf,
                                                              uint32_t n, uint32_t G,
                                                              const uint32_t* __restrict__ group,
                                                              ItsCell* __restrict__ cells) {
    pdl_wait();
    const uint32_t g = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;  // whole warps
    if (g * 32u >= G) return;
    uint32_t hi;
    const uint32_t x = cell_start_warp<false, OWN>(cmf, n, G, group, g, hi);
    const uint32_t k = g * 32u + (threadIdx.x & 31u);
    // the end of a cell is the next cell's start: the next lane's, or the next group's
    uint32_t y = __shfl_down_sync(0xffffffffu, x, 1);
    if ((threadIdx.x & 31u) == 31u) y = hi;
    if (k >= G) return;
    if (k + 1u >= G) y = n - 1u;
    const uint32_t d = cell_part(x, y);
    float v[kCellParts];
#pragma unroll
    for (int j = 0; j < kCellParts; ++j)
        v[j] = __ldg(cmf + min(x + (j + 1) * d - 1u, y));
    uint32_t ym = y;
    if (x > 0u) {
        const float ck = cell_at(cell_step<false>(cmf, n, G), k);
        if (!(x <= n - 1u && __ldg(cmf + x - 1u) < ck)) ym |= kCellUnsafe;
    }
    uint4* dst = reinterpret_cast<uint4*>(cells + k);
    dst[0] = make_uint4(x, ym, __float_as_uint(v[0]), __float_as_uint(v[1]));
    dst[1] = make_uint4(__float_as_uint(v[2]), __float_as_uint(v[3]), __float_as_uint(v[4]),
                        __float_as_uint(v[5]));
}

// ---- the grid of the compensated CMF ------------------------------------------------------

__device__ __forceinline__ uint32_t grid_f(float v, float scale) {
    return __float2uint_rz(__fmul_rn(v, scale));  // (exact product; NaN and negative values: 0)
}

// One cell per lane, a warp per 32 (cell_start_warp finds their starts): the steps of its parts'
// last items.  0.051 ms at n = 2^24 (2^21 cells, 64 MB written, the CMF read once from HBM: 2.6
// TB/s), issue-bound: 27 loads and conversions a cell.
template <bool OWN>
__global__ __launch_bounds__(kSampleThreads) void k_its_grids(const float* __restrict__ cmf,
                                                              uint32_t n, uint32_t G,
                                                              const uint32_t* __restrict__ group,
                                                              ItsGrid* __restrict__ grids) {
    pdl_wait();
    const uint32_t g = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;  // whole warps
    if (g * 32u >= G) return;
    uint32_t hi;
    const uint32_t x = cell_start_warp<true, OWN>(cmf, n, G, group, g, hi);
    const uint32_t k = g * 32u + (threadIdx.x & 31u);
    uint32_t y = __shfl_down_sync(0xffffffffu, x, 1);
    if ((threadIdx.x & 31u) == 31u) y = hi;
    if (k >= G) return;
    if (k + 1u >= G) y = n - 1u;
    const uint32_t m = y > x ? y - x : 0u;  // items of the cell (y itself is the next cell's first)
    uint32_t e = 0;
    while ((static_cast<uint64_t>(kGridSlots) << e) < m) ++e;
    const uint32_t parts = m >> e;  // whole parts (the rest is below y, the next cell's first)
    const float scale = pow2f(its_shift(__ldg(cmf + n - 1u), G));
    uint32_t w[8];
    w[0] = x;
#pragma unroll
    for (int c = 0; c < 7; ++c) {
        uint32_t f[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const uint32_t j = 4u * c + i;
            f[i] = 127u;
            if (j < kGridSlots && j < parts)
                f[i] = grid_f(__ldg(cmf + x + ((j + 1u) << e) - 1u), scale) & 127u;
        }
        w[1 + c] = 0x80808080u | f[0] | f[1] << 8 | f[2] << 16 | f[3] << 24;
    }
    w[7] = (w[7] & 0xffffffu) | e << 24;
    uint4* dst = reinterpret_cast<uint4*>(grids + k);
    dst[0] = make_uint4(w[0], w[1], w[2], w[3]);
    dst[1] = make_uint4(w[4], w[5], w[6], w[7]);
}

// The smallest float that is not below T = (2x + 1) * total * 2^-33: "T > c" for a float c is
// "its_target > c".
__device__ __forceinline__ float its_target(uint32_t x, float total) {
    const uint32_t e = __float_as_uint(total) >> 23;
    if (e >= 67u && e < 255u) {  // total >= 2^-60: every power below is normal
        // total = mt * 2^(e - 150): the 57-bit product rounded up to 24 bits, then scaled exactly
        const uint32_t mt = (__float_as_uint(total) & 0x7fffffu) | 0x800000u;
        const uint64_t P = (static_cast<uint64_t>(x) * mt << 1) + mt;
        return __fmul_rn(__ull2float_ru(P), pow2f(static_cast<int>(e) - 150 - 33));
    }
    float t_hi;
    int t_sgn;
    exact_target(x, total, t_hi, t_sgn);
    return t_sgn > 0 ? __uint_as_float(__float_as_uint(t_hi) + 1u) : t_hi;
}

// Samples per thread: two blocks of 8 words leave room for a full SM of warps.
constexpr int kGridPerThread = 2;

// One 32-byte sector of the grid (2 to 4 bytes per weight at entry 4) settles a sample, with no
// division and no search for its cell.  n = 2^24, 2^26 samples: log-normal 0.97 -> 0.40 ms, uniform
// 0.91 -> 0.34 (195 G/s; issue 72 % active, 145 instructions per 32 samples), against the FP32 cells'
// six values and index range (8 bytes per weight, 332 instructions); n = 2^26, 2^27 samples: uniform
// 2.46 -> 1.10, log-normal 2.78 -> 1.80 ms (the grid exceeds L2: random HBM reads again).
//
// CACHED: a grid that fits the L1s is read through them.  A small one read around them comes from a
// few L2 sectors that every SM asks for: n = 1000 uniform, 2^24 samples 541 us around, 109 through
// (199 by the FP32 cells); n = 10^4 132 and 108, n = 2 * 10^4 (78 KB) 182 and 111.  At 156 KB both take
// 103; a larger one only pushes the CMF values out (64 MB, the shaders' stream, 2^26 samples: 586 and
// 604; n = 10^6 with entry 64, 244 KB, 794 and 829).
constexpr uint32_t kGridCachedMax = 4096;  // cells: 128 KB

template <uint32_t RNG, bool CACHED>
__global__ __launch_bounds__(kSampleThreads) void k_its_sample_grids(
    const float* __restrict__ cmf, uint32_t n, const ItsGrid* __restrict__ grids, uint32_t G,
    uint64_t S, uint64_t seed, uint64_t offset, uint32_t* __restrict__ out) {
    pdl_wait();
    const uint64_t s0 =
        (static_cast<uint64_t>(blockIdx.x) * blockDim.x + threadIdx.x) * kGridPerThread;
    if (s0 >= S) return;
    const uint32_t last = n - 1u;
    const float total = __ldg(cmf + last);
    const float scale = pow2f(its_shift(total, G));
    float t[kGridPerThread];
    if constexpr (RNG == RNG_REF) {
        const uint32_t seed32 = static_cast<uint32_t>(seed);
#pragma unroll
        for (int v = 0; v < kGridPerThread; ++v)
            t[v] = search_range_u(cmf, 0, last,
                                  unit_ref(wang_hash((seed32 ^ 0xA9EC5C80u) +
                                                     static_cast<uint32_t>(offset + s0 + v))));
    } else {
        uint2 ks[10];
        philox4x32_10_keys(seed, ks);
#pragma unroll
        for (int v = 0; v < kGridPerThread; ++v) {
            const uint64_t g = offset + s0 + v;
            const uint4 r = philox4x32_10(
                make_uint4(static_cast<uint32_t>(g), static_cast<uint32_t>(g >> 32), 0u, 0u), ks);
            t[v] = its_target(r.x, total);
        }
    }
    uint4 lo[kGridPerThread], hi[kGridPerThread];
    uint32_t F[kGridPerThread], res[kGridPerThread];
#pragma unroll
    for (int v = 0; v < kGridPerThread; ++v) {
        F[v] = grid_f(t[v], scale);
        const uint32_t* cell = reinterpret_cast<const uint32_t*>(grids + min(F[v] >> 7, G - 1u));
        if constexpr (CACHED)
            ld_u32x8(cell, lo[v], hi[v]);
        else
            ld_block(cell, lo[v], hi[v]);
    }
#pragma unroll
    for (int v = 0; v < kGridPerThread; ++v) {
        // the first part whose last item's step is not below the target's: the steps do not
        // decrease, so the word that holds it is found by its last byte (a word is below the
        // target's step in its last byte exactly when it is below `edge`), the byte in the word
        // by the borrow-free difference of its bytes (stored as 128 + step)
        const uint32_t step = F[v] & 127u, edge = (step | 128u) << 24;
        const uint32_t w6 = hi[v].w | 0xff000000u;
        const bool up = hi[v].x < edge;                       // words 4 .. 6
        const uint32_t mid = up ? hi[v].z : lo[v].z;          // word 5 or 1
        const bool up2 = mid < edge;
        const uint32_t leaf = up ? (up2 ? w6 : hi[v].y) : (up2 ? lo[v].w : lo[v].y);  // 6 4 2 0
        const bool up3 = leaf < edge;
        const uint32_t word = up3 ? (up2 ? (up ? w6 : hi[v].x) : mid) : leaf;
        const uint32_t r = word - step * 0x01010101u;
        const uint32_t ge = r & 0x80808080u;
        const uint32_t in = 4u - __popc(ge);
        const uint32_t below = (up ? 16u : 0u) + (up2 ? 8u : 0u) + (up3 ? 4u : 0u) + in;
        const uint32_t e = hi[v].w >> 24;
        const uint32_t x0 = min(lo[v].x, last);
        uint32_t x = min(x0 + below, last);
        // items in the target's own step are told apart by it from 2^23 steps on
        const bool same = F[v] < (1u << 23) && (r >> (8u * in & 31u) & 0x7fu) == 0u;
        if (e != 0u) {
            const uint64_t end = x0 + (static_cast<uint64_t>(same ? kGridSlots + 1u : below + 1u) << e) - 1u;
            x = static_cast<uint32_t>(min(x0 + (static_cast<uint64_t>(below) << e), static_cast<uint64_t>(last)));
            uint32_t y = static_cast<uint32_t>(min(end, static_cast<uint64_t>(last)));
            while (x < y) {
                const uint32_t mid = x + ((y - x) >> 1);
                if (t[v] > __ldg(cmf + mid))
                    x = mid + 1u;
                else
                    y = mid;
            }
        } else if (same) {
            // (the cell's items end before y on the CMF it was built from; on any other the walk ends)
            const uint32_t y = min(x0 + static_cast<uint32_t>(kGridSlots), last);
            while (x < y && t[v] > __ldg(cmf + x)) ++x;
        }
        res[v] = x;
    }
    if (s0 + kGridPerThread <= S && (reinterpret_cast<uintptr_t>(out) & 7u) == 0) {
        __stcs(reinterpret_cast<uint2*>(out + s0), make_uint2(res[0], res[1]));
    } else {
#pragma unroll
        for (int v = 0; v < kGridPerThread; ++v)
            if (s0 + v < S) __stcs(out + s0 + v, res[v]);
    }
}

// ---- cells on an FP32 CMF: cells whose targets can meet an inversion ------------------
//
// On a CMF that is not monotone every lower-bound search still returns the bisection's index
// for a target t that lies in no inversion interval (cmf[j], cmf[i]] (i < j, cmf[j] < cmf[i]):
// then every value below t comes before every value >= t.  For each i the union of its
// intervals is (S(i + 1), cmf[i]] with S the suffix minimum, so a pass over the CMF marks the
// cells whose target range meets one (bit 31 of the cell's y; n < 2^31), and the cells whose
// start x does not have cmf[x - 1] < c_k; a CMF with a value that is not finite or is negative
// marks every cell.  The cell search serves the unmarked cells and the bisection the others.
constexpr uint32_t kMarkSpan = 64;  // an interval over more cells marks the whole CMF unsafe

// the largest k < G with c_k = fl(step * k) < t (0 if none): the cell of targets just above t
__device__ __forceinline__ uint32_t cell_below(float t, float step, uint32_t G) {
    uint32_t lo = 0, hi = G - 1u;  // c_0 = 0
    while (lo < hi) {
        const uint32_t mid = lo + ((hi - lo + 1u) >> 1);
        if (__fmul_rn(step, __uint2float_rn(mid)) < t)
            lo = mid;
        else
            hi = mid - 1u;
    }
    return lo;
}

// per 4096-value tile of the CMF: its minimum; any value that is NaN, infinite or negative
// raises `bad`
__global__ __launch_bounds__(kSampleThreads) void k_cmf_tile_min(const float* __restrict__ cmf,
                                                                 uint32_t n,
                                                                 float* __restrict__ tile_min,
                                                                 uint32_t* __restrict__ bad) {
    pdl_wait();
    __shared__ float s_m[kSampleThreads / 32];
    const uint64_t base = static_cast<uint64_t>(blockIdx.x) * kTileItems;
    float m = INFINITY;
    bool b = false;
    for (uint32_t e = threadIdx.x; e < kTileItems; e += blockDim.x) {
        if (base + e < n) {
            const float v = __ldg(cmf + base + e);
            b = b || !(v >= 0.0f && v <= 3.402823466e38f);
            m = fminf(m, v);
        }
    }
    if (__syncthreads_or(b) && threadIdx.x == 0) atomicOr(bad, 1u);
#pragma unroll
    for (int d = 16; d > 0; d >>= 1) m = fminf(m, __shfl_xor_sync(0xffffffffu, m, d));
    if ((threadIdx.x & 31u) == 0) s_m[threadIdx.x >> 5] = m;
    __syncthreads();
    if (threadIdx.x == 0) {
        for (int w = 1; w < static_cast<int>(kSampleThreads / 32); ++w) m = fminf(m, s_m[w]);
        tile_min[blockIdx.x] = fminf(m, s_m[0]);
    }
}

// suffix minima of the tile minima (one CTA, chunks of 1024 from the end)
__global__ __launch_bounds__(1024) void k_tile_suffix_min(const float* __restrict__ tile_min,
                                                          uint32_t tiles,
                                                          float* __restrict__ suf) {
    pdl_wait();
    __shared__ float s_w[32];
    __shared__ float s_carry;
    if (threadIdx.x == 0) s_carry = INFINITY;
    __syncthreads();
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    for (int64_t end = tiles; end > 0; end -= 1024) {
        // thread j holds tile end - 1 - j (reversed, so an inclusive prefix min is a suffix min)
        const int64_t t = end - 1 - static_cast<int64_t>(threadIdx.x);
        float v = t >= 0 ? tile_min[t] : INFINITY;
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
            const float o = __shfl_up_sync(0xffffffffu, v, d);
            if (lane >= d) v = fminf(v, o);
        }
        if (lane == 31) s_w[warp] = v;
        __syncthreads();
        if (warp == 0) {
            float u = s_w[lane];
#pragma unroll
            for (int d = 1; d < 32; d <<= 1) {
                const float o = __shfl_up_sync(0xffffffffu, u, d);
                if (lane >= d) u = fminf(u, o);
            }
            s_w[lane] = u;  // inclusive over warps 0 .. lane
        }
        __syncthreads();
        const float carry = s_carry;
        const float r = fminf(fminf(v, warp ? s_w[warp - 1] : INFINITY), carry);
        if (t >= 0) suf[t] = r;
        __syncthreads();
        if (threadIdx.x == 1023) s_carry = r;
        __syncthreads();
    }
}

// marks the cells k in [cell_below(lo+), cell_below(hi)] for the interval (lo, hi]; an interval
// over more than kMarkSpan cells raises `bad` instead
__device__ __forceinline__ void mark_interval(float lo, float hi, float step, uint32_t G,
                                              ItsCell* __restrict__ cells,
                                              uint32_t* __restrict__ bad) {
    const uint32_t a = cell_below(__uint_as_float(__float_as_uint(lo) + 1u), step, G);
    const uint32_t b = cell_below(hi, step, G);
    if (b >= a && b - a >= kMarkSpan) {
        atomicOr(bad, 1u);
        return;
    }
    for (uint32_t k = a; k <= b; ++k) atomicOr(&cells[k].y, kCellUnsafe);
}

// one CTA per 4096-value tile, 16 consecutive values per thread: S(i + 1) from the thread's own
// later values, the later threads' and the later tiles' minima; every i with S(i + 1) < cmf[i]
// marks the cells of (S(i + 1), cmf[i]].  Skipped when `bad` is set (every cell is marked then).
__global__ __launch_bounds__(kSampleThreads) void k_cmf_mark(const float* __restrict__ cmf,
                                                             uint32_t n, uint32_t G,
                                                             const float* __restrict__ suf,
                                                             uint32_t tiles,
                                                             ItsCell* __restrict__ cells,
                                                             uint32_t* __restrict__ bad) {
    pdl_wait();
    __shared__ float s_w[kSampleThreads / 32];
    // one decision for the whole CTA (other CTAs may raise `bad` meanwhile)
    if (__syncthreads_or(*reinterpret_cast<volatile uint32_t*>(bad) != 0u)) return;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const uint64_t base = static_cast<uint64_t>(blockIdx.x) * kTileItems + threadIdx.x * 16u;
    float v[16];
#pragma unroll
    for (int c = 0; c < 16; ++c) v[c] = base + c < n ? __ldg(cmf + base + c) : INFINITY;
    float tmin = v[15];
#pragma unroll
    for (int c = 14; c >= 0; --c) tmin = fminf(tmin, v[c]);
    // minimum over the later threads of the tile (exclusive), then over the later tiles
    float inc = tmin;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
        const float o = __shfl_down_sync(0xffffffffu, inc, d);
        if (lane + d < 32) inc = fminf(inc, o);
    }
    if (lane == 0) s_w[warp] = inc;  // warp's minimum
    __syncthreads();
    float after = __shfl_down_sync(0xffffffffu, inc, 1);
    if (lane == 31) after = INFINITY;
    for (int w = warp + 1; w < static_cast<int>(kSampleThreads / 32); ++w) after = fminf(after, s_w[w]);
    if (blockIdx.x + 1u < tiles) after = fminf(after, suf[blockIdx.x + 1u]);
    const float step = __fdiv_rn(__ldg(cmf + n - 1u), __uint2float_rn(G));
    float s = after;  // S(i + 1) for the thread's last value
#pragma unroll
    for (int c = 15; c >= 0; --c) {
        if (base + c < n && s < v[c]) mark_interval(s, v[c], step, G, cells, bad);
        s = fminf(s, v[c]);
    }
}

// with `bad` raised (a value that is not finite or is negative, or an interval over too many
// cells) every cell is marked
__global__ __launch_bounds__(kSampleThreads) void k_cells_mark_all(uint32_t G,
                                                                   ItsCell* __restrict__ cells,
                                                                   const uint32_t* __restrict__ bad) {
    pdl_wait();
    if (*reinterpret_cast<const volatile uint32_t*>(bad) == 0u) return;
    for (uint32_t k = blockIdx.x * blockDim.x + threadIdx.x; k < G; k += gridDim.x * blockDim.x)
        cells[k].y |= kCellUnsafe;
}

// The bisection of [0, n - 1] for target t (a probe c sends it right when t > c) through the
// stored probe-tree blocks (L = its_tree_stored_levels(n) > 0 levels: the node alone above the
// last one, whose slot 7 gives the range), then the CMF for the tail: the same probe sequence.
__device__ uint32_t bisect_blocks(const float* __restrict__ cmf, uint32_t n,
                                  const TreeBlock* __restrict__ blocks, uint32_t L, float t) {
    uint32_t node = 1, level = 0, x = 0, y = 0;
    const TreeBlock* lb = blocks;
    for (uint32_t bl = 0; bl < L; ++bl, level += kTreeBlockLevels) {
        const uint32_t first = 1u << level;
        uint4 lo, hi;
        ld_u32x8(reinterpret_cast<const uint32_t*>(lb + (node - first)), lo, hi);
        lb += first;
        const uint32_t r0 = t > __uint_as_float(lo.x) ? 1u : 0u;
        const uint32_t c1 = r0 ? lo.z : lo.y;
        const uint32_t r1 = t > __uint_as_float(c1) ? 1u : 0u;
        const uint32_t c2 = r0 ? (r1 ? hi.z : hi.y) : (r1 ? hi.x : lo.w);
        const uint32_t r2 = t > __uint_as_float(c2) ? 1u : 0u;
        if (bl + 1u < L) {
            node = 8u * node + 4u * r0 + 2u * r1 + r2;
        } else {
            x = hi.w & 0x7fffffffu;
            y = x + (n >> level) + (hi.w >> 31) - 1u;
            const uint32_t r[3] = {r0, r1, r2};
#pragma unroll
            for (int d = 0; d < 3; ++d) {
                const uint32_t mid = x + ((y - x) >> 1);
                x = r[d] ? mid + 1u : x;
                y = r[d] ? y : mid;
            }
            y = min(y, n - 1u);
            x = min(x, y);
        }
    }
    while (x < y) {
        const uint32_t mid = x + ((y - x) >> 1);
        if (t > __ldg(cmf + mid))
            x = mid + 1u;
        else
            y = mid;
    }
    return x;
}

// steps of the cell correction (beyond them the bracket check sends the sample to the
// bisection, so the bound only caps the work)
constexpr int kCellFix = 8;

template <uint32_t RNG>
__global__ __launch_bounds__(kSampleThreads) void k_its_sample_cells(
    const float* __restrict__ cmf, uint32_t n, const ItsCell* __restrict__ cells, uint32_t G,
    uint64_t S, uint64_t seed, uint64_t offset, uint32_t* __restrict__ out,
    const TreeBlock* __restrict__ blocks, uint32_t L) {
    pdl_wait();
    const uint64_t s = static_cast<uint64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
    if (s >= S) return;
    const uint32_t last = n - 1u;
    const float total = __ldg(cmf + last);
    const uint64_t g = offset + s;
    float t_hi;
    int t_sgn = 0;
    if constexpr (RNG == RNG_REF) {
        const uint32_t seed32 = static_cast<uint32_t>(seed);
        t_hi = search_range_u(cmf, 0, last,
                              unit_ref(wang_hash((seed32 ^ 0xA9EC5C80u) + static_cast<uint32_t>(g))));
    } else {
        uint2 ks[10];
        philox4x32_10_keys(seed, ks);
        const uint4 r = philox4x32_10(
            make_uint4(static_cast<uint32_t>(g), static_cast<uint32_t>(g >> 32), 0u, 0u), ks);
        exact_target(r.x, total, t_hi, t_sgn);
    }
    // "T > c" for the target T = (t_hi, t_sgn) (RNG_REF: t_sgn = 0, the shader's u > cmf[mid])
    auto above = [&](float c) { return t_hi > c || (t_hi == c && t_sgn > 0); };
    // the cell holding T: c_k < T <= c_{k+1} with the build's c_k = fl(step * k), from an FP32
    // estimate (off by a few cells at most) moved by exact comparisons
    const float step = __fdiv_rn(total, __uint2float_rn(G));
    const float scale = __fdiv_rn(__uint2float_rn(G), total);
    uint32_t k = __float2uint_rz(__fmul_rn(t_hi, scale));
    k = k < G - 1u ? k : G - 1u;
    for (int it = 0; it < kCellFix && k > 0u && !above(__fmul_rn(step, __uint2float_rn(k))); ++it)
        --k;
    for (int it = 0; it < kCellFix && k + 1u < G && above(__fmul_rn(step, __uint2float_rn(k + 1u)));
         ++it)
        ++k;
    // c_k < T <= c_{k+1} (then cmf[x_k - 1] < c_k < T, and T is in the range the cell's
    // inversion mark covers); cmf[y_k] >= T is checked on the block
    const bool settled = (k == 0u || above(__fmul_rn(step, __uint2float_rn(k)))) &&
                         (k + 1u >= G || !above(__fmul_rn(step, __uint2float_rn(k + 1u))));
    const uint64_t once = l2_policy_evict_first();
    uint4 q0, q1;
    ld_u32x8_policy(reinterpret_cast<const uint32_t*>(cells + k), once, q0, q1);
    // an FP32 CMF's cell may be marked (its targets can meet an inversion, or its start is not
    // below c_k): bisect those
    const bool unsafe = (q0.y & kCellUnsafe) != 0u;
    // (a cell block holds indices < n for the n it was built for; the clamp keeps any other
    // block's search inside the CMF)
    uint32_t x = q0.x, y = min(q0.y & ~kCellUnsafe, last);
    const float v[kCellParts] = {__uint_as_float(q0.z), __uint_as_float(q0.w),
                                 __uint_as_float(q1.x), __uint_as_float(q1.y),
                                 __uint_as_float(q1.z), __uint_as_float(q1.w)};
    // (y >= x holds for every non-decreasing CMF; the test keeps weights outside the
    // contract -- NaN, negative -- from producing an index outside [0, N))
    if (!unsafe && settled && y >= x && !above(v[kCellParts - 1])) {
        // the first part whose last value is >= T (the values are non-decreasing)
        uint32_t part = 0;
#pragma unroll
        for (int j = 0; j < kCellParts; ++j) part += above(v[j]) ? 1u : 0u;
        const uint32_t d = cell_part(x, y);
        const uint32_t lo = x + part * d;
        if (d == 1u) {
            __stcs(out + s, lo);
            return;
        }
        y = min(lo + d - 1u, y);  // cmf[y] >= T and cmf[lo - 1] < T
        x = lo;
    } else if (blocks) {
        // the bisection through the stored probe tree (t_hi with the tie folded in: T > c
        // exactly when the next float above t_hi is > c, for t_sgn > 0)
        const float t = t_sgn > 0 ? __uint_as_float(__float_as_uint(t_hi) + 1u) : t_hi;
        __stcs(out + s, bisect_blocks(cmf, n, blocks, L, t));
        return;
    } else {
        x = 0;
        y = last;
    }
    while (x < y) {
        const uint32_t mid = x + ((y - x) >> 1);
        if (above(ld_f32_policy(cmf + mid, once)))
            x = mid + 1;
        else
            y = mid;
    }
    __stcs(out + s, x);
}

// Guiding table of an exactly non-decreasing CMF: the same entries as k_cutpoint_guide
// (guide[k] = lower bound of fl(fl(total / G) * k), clamped to N - 1), where every lower-bound
// search gives the same index, so the bracketed searches of cell_start apply.
template <bool OWN>
__global__ __launch_bounds__(kSampleThreads) void k_guide_monotone(const float* __restrict__ cmf,
                                                                   uint32_t n, uint32_t G,
                                                                   const uint32_t* __restrict__ group,
                                                                   uint32_t* __restrict__ guide) {
    pdl_wait();
    const uint32_t g = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;  // whole warps
    if (g * 32u >= G) return;
    uint32_t hi;
    const uint32_t x = cell_start_warp<false, OWN>(cmf, n, G, group, g, hi);
    const uint32_t k = g * 32u + (threadIdx.x & 31u);
    if (k < G) guide[k] = x;
}

// Up to this many cells the second pass's warps find their brackets themselves: a launch less, and
// few enough warps that all wait at once.  Builds, with the first pass / without: ITS n = 65536 (8192
// cells) 18.6 / 16.7 us, n = 5000 14.8 / 13.9, n = 262144 (32768) 19.6 / 17.4; Cutpoint, entry 32, n = 10^5
// (3125) 18.1 / 16.9, n = 10^6 (31250) 23.3 / 21.3.  The line is where both met when kernels still let their
// dependents start early; since then n = 2^22 (131072) takes 34.6 / 32.3, so it is on the safe side.
constexpr uint32_t kOwnMaxCells = 32768;

// the first pass (group: group_entries(G) words); true: left to the second
template <bool GRID>
static bool launch_cell_groups(cudaStream_t st, const float* cmf, uint32_t n, uint32_t G,
                               uint32_t* group) {
    if (G <= kOwnMaxCells) return true;
    launch_pdl(k_cell_groups<GRID>, (group_entries(G) + kSampleThreads - 1) / kSampleThreads,
               kSampleThreads, 0, st, cmf, n, G, group);
    return false;
}

static uint32_t warp_blocks(uint32_t G) {
    const uint64_t threads = (static_cast<uint64_t>(G) + 31u) / 32u * 32u;
    return static_cast<uint32_t>((threads + kSampleThreads - 1) / kSampleThreads);
}

cudaError_t launch_its_cells(cudaStream_t st, const float* cmf, uint32_t n, uint32_t G,
                             uint32_t* group, ItsCell* cells) {
    const bool own = launch_cell_groups<false>(st, cmf, n, G, group);
    launch_pdl(own ? k_its_cells<true> : k_its_cells<false>, warp_blocks(G), kSampleThreads, 0, st, cmf, n, G, group, cells);
    return cudaGetLastError();
}

cudaError_t launch_its_grids(cudaStream_t st, const float* cmf, uint32_t n, uint32_t G,
                             uint32_t* group, ItsGrid* grids) {
    const bool own = launch_cell_groups<true>(st, cmf, n, G, group);
    launch_pdl(own ? k_its_grids<true> : k_its_grids<false>, warp_blocks(G), kSampleThreads, 0, st, cmf, n, G, group, grids);
    return cudaGetLastError();
}

cudaError_t launch_its_sample_grids(cudaStream_t st, uint32_t rng, const float* cmf, uint32_t n,
                                    const ItsGrid* grids, uint32_t G, uint64_t S, uint64_t seed,
                                    uint64_t offset, uint32_t* out) {
    constexpr uint64_t per = kSampleThreads * kGridPerThread;
    const uint64_t grid = (S + per - 1) / per;
    if (grid == 0) return cudaSuccess;
    if (grid > 0x7fffffffull) return cudaErrorInvalidValue;
    const bool cached = G <= kGridCachedMax;
    auto go = [&](auto kernel) {
        launch_pdl(kernel, static_cast<unsigned>(grid), kSampleThreads, 0, st, cmf, n, grids, G, S, seed,
                   offset, out);
    };
    if (rng == RNG_REF)
        cached ? go(k_its_sample_grids<RNG_REF, true>) : go(k_its_sample_grids<RNG_REF, false>);
    else
        cached ? go(k_its_sample_grids<RNG_PHILOX, true>) : go(k_its_sample_grids<RNG_PHILOX, false>);
    return cudaGetLastError();
}

cudaError_t launch_its_marks(cudaStream_t st, const float* cmf, uint32_t n, uint32_t G,
                             ItsCell* cells, float* tile_scratch, uint32_t* bad) {
    const uint32_t tiles = tiles_for(n);
    float* tile_min = tile_scratch;
    float* suf = tile_scratch + tiles;
    cudaError_t e = cudaMemsetAsync(bad, 0, sizeof(uint32_t), st);
    if (e != cudaSuccess) return e;
    launch_pdl(k_cmf_tile_min, tiles, kSampleThreads, 0, st, cmf, n, tile_min, bad);
    launch_pdl(k_tile_suffix_min, 1, 1024, 0, st, tile_min, tiles, suf);
    launch_pdl(k_cmf_mark, tiles, kSampleThreads, 0, st, cmf, n, G, suf, tiles, cells, bad);
    // (a grid-stride loop: any grid covers the cells; most launches return at once)
    const uint32_t mark_grid = min((G + kSampleThreads - 1) / kSampleThreads, 1024u);
    launch_pdl(k_cells_mark_all, mark_grid, kSampleThreads, 0, st, G, cells, bad);
    return cudaGetLastError();
}

cudaError_t launch_its_sample_cells(cudaStream_t st, uint32_t rng, const float* cmf, uint32_t n,
                                    const ItsCell* cells, uint32_t G, uint64_t S, uint64_t seed,
                                    uint64_t offset, uint32_t* out, const TreeBlock* blocks,
                                    uint32_t L) {
    const uint64_t grid = (S + kSampleThreads - 1) / kSampleThreads;
    if (grid == 0) return cudaSuccess;
    if (grid > 0x7fffffffull) return cudaErrorInvalidValue;
    if (rng == RNG_REF)
        launch_pdl(k_its_sample_cells<RNG_REF>, static_cast<unsigned>(grid), kSampleThreads, 0, st, 
            cmf, n, cells, G, S, seed, offset, out, blocks, L);
    else
        launch_pdl(k_its_sample_cells<RNG_PHILOX>, static_cast<unsigned>(grid), kSampleThreads, 0, st, 
            cmf, n, cells, G, S, seed, offset, out, blocks, L);
    return cudaGetLastError();
}

// ---- Cutpoint (guiding table) -----------------------------------------------------------

// cutpoint/guiding_table/shader.comp:40-55: entry k = lower bound of (total / G) * k over the
// whole CMF, with the shader's FP32 step and probe sequence.
__global__ __launch_bounds__(kSampleThreads) void k_cutpoint_guide(const float* __restrict__ cmf,
                                                                   uint32_t n, uint32_t G,
                                                                   uint32_t* __restrict__ guide) {
    pdl_wait();
    const uint32_t k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= G) return;
    const float total = __ldg(cmf + n - 1u);
    const float step = __fdiv_rn(total, __uint2float_rn(G));
    guide[k] = bisect(cmf, 0, n - 1u, __fmul_rn(step, __uint2float_rn(k)));
}

// cutpoint/sampling/shader.comp:100-140.  The subgroup's elected lane (the first sample of the
// aligned group of 32) draws u1, which picks guiding cell k = min(u1 * G, G - 1); the search
// range is [guide[k], guide[k + 1]] (up to N - 1 for the last cell), and every sample bisects
// it for u2 drawn inside the cell's CMF range.  RNG_REF: u1 = wang_hash(seed + g0), u2 =
// wang_hash((seed ^ 0x79145147) + g) as the shader; RNG_PHILOX: u1 = x0 of the group's first
// sample, u2 = x1 of the sample (Philox4x32-10, counter = sample index).
template <uint32_t RNG>
__global__ __launch_bounds__(kSampleThreads) void k_cutpoint_sample(
    const float* __restrict__ cmf, uint32_t n, const uint32_t* __restrict__ guide, uint32_t G,
    uint64_t S, uint64_t seed, uint64_t offset, uint32_t* __restrict__ out) {
    pdl_wait();
    const uint64_t s = static_cast<uint64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
    if (s >= S) return;
    const uint64_t g = offset + s, g0 = offset + (s & ~31ull);
    float u1, uu;
    if constexpr (RNG == RNG_REF) {
        const uint32_t seed32 = static_cast<uint32_t>(seed);
        u1 = unit_ref(wang_hash(seed32 + static_cast<uint32_t>(g0)));
        uu = unit_ref(wang_hash((seed32 ^ 0x79145147u) + static_cast<uint32_t>(g)));
    } else {
        uint2 ks[10];
        philox4x32_10_keys(seed, ks);
        const uint4 r0 = philox4x32_10(
            make_uint4(static_cast<uint32_t>(g0), static_cast<uint32_t>(g0 >> 32), 0u, 0u), ks);
        const uint4 r = philox4x32_10(
            make_uint4(static_cast<uint32_t>(g), static_cast<uint32_t>(g >> 32), 0u, 0u), ks);
        u1 = unit_ref(r0.x);
        uu = unit_ref(r.y);
    }
    uint32_t k = __float2uint_rz(__fmul_rn(u1, __uint2float_rn(G)));
    k = k < G - 1u ? k : G - 1u;
    // (entries are < n for the CMF the table was built from; the clamps keep a table built
    // for another n from reading outside the CMF)
    const uint32_t x = min(__ldg(guide + k), n - 1u);
    const uint32_t y = k != G - 1u ? max(min(__ldg(guide + k + 1u), n - 1u), x) : n - 1u;
    const float u2 = search_range_u(cmf, x, y, uu);
    __stcs(out + s, bisect(cmf, x, y, u2));
}

// The same samples on a CMF that does not decrease, where the bisection's index is x plus the number
// of the range's values below u2.  A warp takes kCutGroups groups: its first lanes find the groups'
// ranges (u1, guiding entries, ends) once, through shared memory; then, group by group, the lanes
// hold the range's values, R consecutive ones each, and every lane counts through shuffles: a search
// over the lanes' last values, then the R - 1 values before it.  Instruction issue bounds it (84 %
// active; 71 instructions per 32 samples, the per-sample bisection took 137 and found its range 32
// times): entry 32, n = 2^22, 2^26 samples: uniform, the shaders' stream 0.315 -> 0.147 ms; log-normal,
// Philox 0.486 -> 0.263 (4 groups a warp 0.207 / 0.361 before the loop was unrolled, 8 0.187 / 0.326).
constexpr int kCutGroups = 8;
// fewer samples leave SMs without a warp of kCutGroups groups: 10^6 samples (n = 10^6) 13.3 us by
// the bisection, 12.4 by groups; 7 x 10^4 (n = 5000) 11.1 and 13.1
constexpr uint64_t kCutMonoMin = 1u << 19;

// # of values below t; v[r] of lane l = value R l + r of the range, +inf past its end (at most
// 32 R - 1 values, so the last lane's last is)
template <int R>
__device__ __forceinline__ uint32_t count_below(const float (&v)[R], float t) {
    uint32_t c = 0;
#pragma unroll
    for (uint32_t st = 16; st > 0; st >>= 1)
        c += __shfl_sync(0xffffffffu, v[R - 1], c + st - 1u) < t ? st : 0u;
    uint32_t in = 0;
#pragma unroll
    for (int r = 0; r + 1 < R; ++r) in += __shfl_sync(0xffffffffu, v[r], c) < t ? 1u : 0u;
    return R * c + in;
}
template <int R>
__device__ __forceinline__ uint32_t range_count(const float* __restrict__ cmf, uint32_t x, uint32_t m,
                                                uint32_t lane, float t) {
    float v[R];
    const float* const at = cmf + x + R * lane;
#pragma unroll
    for (int r = 0; r < R; ++r) v[r] = R * lane + r < m ? __ldg(at + r) : __int_as_float(0x7f800000);
    return count_below<R>(v, t);
}

template <uint32_t RNG>
__global__ __launch_bounds__(kSampleThreads) void k_cutpoint_sample_mono(
    const float* __restrict__ cmf, uint32_t n, const uint32_t* __restrict__ guide, uint32_t G,
    uint64_t S, uint64_t seed, uint64_t offset, uint32_t* __restrict__ out) {
    pdl_wait();
    __shared__ uint4 s_range[kSampleThreads / 32][kCutGroups];
    const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31u;
    const uint64_t base = (static_cast<uint64_t>(blockIdx.x) * (kSampleThreads / 32) + warp) * (kCutGroups * 32u);
    if (base >= S) return;  // whole warps
    uint2 ks[10];
    if constexpr (RNG == RNG_PHILOX) philox4x32_10_keys(seed, ks);
    const uint32_t seed32 = static_cast<uint32_t>(seed);
    if (lane < kCutGroups) {
        const uint64_t g0 = offset + base + lane * 32u;
        float u1;
        if constexpr (RNG == RNG_REF)
            u1 = unit_ref(wang_hash(seed32 + static_cast<uint32_t>(g0)));
        else
            u1 = unit_ref(philox4x32_10(make_uint4(static_cast<uint32_t>(g0),
                                                   static_cast<uint32_t>(g0 >> 32), 0u, 0u), ks).x);
        uint32_t k = __float2uint_rz(__fmul_rn(u1, __uint2float_rn(G)));
        k = k < G - 1u ? k : G - 1u;
        const uint32_t x = min(__ldg(guide + k), n - 1u);
        const uint32_t y = k != G - 1u ? max(min(__ldg(guide + k + 1u), n - 1u), x) : n - 1u;
        const float lo = x > 0 ? __ldg(cmf + x - 1) : 0.0f;
        s_range[warp][lane] = make_uint4(x, y - x, __float_as_uint(lo),
                                         __float_as_uint(__fsub_rn(__ldg(cmf + y), lo)));
    }
    __syncwarp();
    // the index drawn by this lane's sample of group p
    const uint32_t c0 = static_cast<uint32_t>(offset + base) + lane;
    auto draw = [&](int p) -> uint32_t {
        const uint4 range = s_range[warp][p];
        float uu;
        if constexpr (RNG == RNG_REF) {
            uu = unit_ref(wang_hash((seed32 ^ 0x79145147u) + (c0 + 32u * p)));
        } else {
            const uint64_t g = offset + base + (lane + 32u * p);
            uu = unit_ref(philox4x32_10(make_uint4(static_cast<uint32_t>(g),
                                                   static_cast<uint32_t>(g >> 32), 0u, 0u), ks).y);
        }
        const float u2 = __fadd_rn(__uint_as_float(range.z), __fmul_rn(__uint_as_float(range.w), uu));
        const uint32_t x = range.x, m = range.y;
        if (m < 64u) return x + range_count<2>(cmf, x, m, lane, u2);
        if (m < 256u) return x + range_count<8>(cmf, x, m, lane, u2);
        return bisect(cmf, x, x + m, u2);
    };
    uint32_t* const dst = out + base + lane;
    if (base + kCutGroups * 32u <= S) {
#pragma unroll
        for (int p = 0; p < kCutGroups; ++p) __stcs(dst + 32 * p, draw(p));
    } else {
#pragma unroll 1
        for (int p = 0; p < kCutGroups && base + p * 32u < S; ++p) {
            const uint32_t i = draw(p);
            if (base + p * 32u + lane < S) __stcs(dst + 32 * p, i);
        }
    }
}

cudaError_t launch_cutpoint_guide(cudaStream_t st, const float* cmf, uint32_t n, uint32_t G,
                                  uint32_t* guide) {
    const uint32_t blocks = (G + kSampleThreads - 1) / kSampleThreads;
    launch_pdl(k_cutpoint_guide, blocks, kSampleThreads, 0, st, cmf, n, G, guide);
    return cudaGetLastError();
}

cudaError_t launch_guide_monotone(cudaStream_t st, const float* cmf, uint32_t n, uint32_t G,
                                  uint32_t* group, uint32_t* guide) {
    const bool own = launch_cell_groups<false>(st, cmf, n, G, group);
    launch_pdl(own ? k_guide_monotone<true> : k_guide_monotone<false>, warp_blocks(G), kSampleThreads, 0, st, cmf, n, G, group, guide);
    return cudaGetLastError();
}

cudaError_t launch_cutpoint_sample(cudaStream_t st, uint32_t rng, const float* cmf, uint32_t n,
                                   const uint32_t* guide, uint32_t G, uint64_t S, uint64_t seed,
                                   uint64_t offset, uint32_t* out, bool monotone) {
    monotone = monotone && S >= kCutMonoMin;
    const uint64_t per = monotone ? kSampleThreads * kCutGroups : kSampleThreads;
    const uint64_t blocks = (S + per - 1) / per;
    if (blocks == 0) return cudaSuccess;
    if (blocks > 0x7fffffffull) return cudaErrorInvalidValue;
    if (monotone) {
        if (rng == RNG_REF)
            launch_pdl(k_cutpoint_sample_mono<RNG_REF>, static_cast<unsigned>(blocks), kSampleThreads,
                       0, st, cmf, n, guide, G, S, seed, offset, out);
        else
            launch_pdl(k_cutpoint_sample_mono<RNG_PHILOX>, static_cast<unsigned>(blocks),
                       kSampleThreads, 0, st, cmf, n, guide, G, S, seed, offset, out);
        return cudaGetLastError();
    }
    if (rng == RNG_REF)
        launch_pdl(k_cutpoint_sample<RNG_REF>, static_cast<unsigned>(blocks), kSampleThreads, 0, st, 
            cmf, n, guide, G, S, seed, offset, out);
    else
        launch_pdl(k_cutpoint_sample<RNG_PHILOX>, static_cast<unsigned>(blocks), kSampleThreads, 0, st, 
            cmf, n, guide, G, S, seed, offset, out);
    return cudaGetLastError();
}

cudaError_t launch_alias_sample(cudaStream_t st, uint32_t rng, uint32_t coop, const uint2* table,
                                const AliasBlock* blocks, const unsigned long long* reads,
                                uint32_t n, uint64_t S, uint64_t seed, uint64_t offset,
                                uint32_t* out) {
    const bool b = blocks && reads && !coop;  // cooperative: the table alone
    const uint64_t per = b ? kBlockPerThread : kAliasPerThread;
    const uint64_t threads = (S + per - 1) / per;
    const uint64_t ctas = (threads + kSampleThreads - 1) / kSampleThreads;
    if (ctas == 0) return cudaSuccess;
    if (ctas > 0x7fffffffull) return cudaErrorInvalidValue;
    const dim3 grid(static_cast<unsigned>(ctas));
    auto go = [&](auto kernel) {
        launch_pdl(kernel, grid, kSampleThreads, 0, st, table, blocks, reads, n, S, seed, offset, coop, out);
    };
    if (rng == RNG_REF) {
        if (coop)
            go(k_alias_sample<RNG_REF, true, false>);
        else if (b)
            go(k_alias_sample<RNG_REF, false, true>);
        else
            go(k_alias_sample<RNG_REF, false, false>);
    } else if (b) {
        go(k_alias_sample<RNG_PHILOX, false, true>);
    } else {
        go(k_alias_sample<RNG_PHILOX, false, false>);
    }
    return cudaGetLastError();
}

cudaError_t launch_alias_blocks(cudaStream_t st, const uint2* table, const uint32_t* classes,
                                uint32_t n, AliasBlock* blocks, unsigned long long* reads) {
    constexpr uint32_t span = kBlockBuildThreads * 32u;  // entries per CTA
    launch_pdl(k_alias_blocks, static_cast<unsigned>((static_cast<uint64_t>(n) + span - 1) / span),
               kBlockBuildThreads, 0, st, table, classes, n, blocks, reads);
    return cudaGetLastError();
}

cudaError_t launch_batch_alias_sample(cudaStream_t st, uint32_t rng, uint32_t coop,
                                      const BatchView& b) {
    if (b.sample_blocks == 0) return cudaSuccess;
    auto go = [&](auto kernel, uint32_t c) {
        launch_pdl(kernel, b.sample_blocks, kSampleThreads, 0, st, b, c);
    };
    if (rng == RNG_REF) {
        if (coop)
            go(k_alias_sample_batch<RNG_REF, true>, coop);
        else
            go(k_alias_sample_batch<RNG_REF, false>, 0u);
    } else {
        go(k_alias_sample_batch<RNG_PHILOX, false>, 0u);
    }
    return cudaGetLastError();
}

cudaError_t launch_its_tree(cudaStream_t st, const float* cmf, uint32_t n, uint32_t L,
                            TreeBlock* blocks) {
    const size_t count = its_tree_blocks(L);
    if (count == 0) return cudaSuccess;
    const size_t grid = (count + kSampleThreads - 1) / kSampleThreads;
    if (grid > 0x7fffffffull) return cudaErrorInvalidValue;
    launch_pdl(k_its_tree, static_cast<unsigned>(grid), kSampleThreads, 0, st, cmf, n, L, blocks);
    return cudaGetLastError();
}

cudaError_t launch_its_sample(cudaStream_t st, uint32_t rng, uint32_t coop, bool parray,
                              const float* cmf, uint32_t n, uint64_t S, uint64_t seed,
                              uint64_t offset, uint32_t* out, const TreeBlock* tree,
                              uint32_t B) {
    const uint64_t blocks = (S + kSampleThreads - 1) / kSampleThreads;
    if (blocks == 0) return cudaSuccess;
    if (blocks > 0x7fffffffull) return cudaErrorInvalidValue;
    const dim3 grid(static_cast<unsigned>(blocks));
    if (coop == 0) {
        const uint64_t groups = (S + kItsGroup - 1) / kItsGroup;
        const unsigned tb = static_cast<unsigned>(groups < kItsMaxBlocks ? groups : kItsMaxBlocks);
        if (rng == RNG_REF)
            launch_pdl(k_its_sample_tree<RNG_REF>, tb, kSampleThreads, 0, st, cmf, n, S, seed, offset, out,
                                                                      tree, B);
        else
            launch_pdl(k_its_sample_tree<RNG_PHILOX>, tb, kSampleThreads, 0, st, cmf, n, S, seed, offset,
                                                                         out, tree, B);
    } else if (parray) {
        launch_pdl(k_its_sample<RNG_REF, 2>, grid, kSampleThreads, 0, st, cmf, n, S, seed, offset, coop, out);
    } else {
        launch_pdl(k_its_sample<RNG_REF, 1>, grid, kSampleThreads, 0, st, cmf, n, S, seed, offset, coop, out);
    }
    return cudaGetLastError();
}

}  // namespace wrs
