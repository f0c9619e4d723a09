// sm_100a kernels of the candidate-key search path.
//
//   k_build_table  fills the comb table in HBM: entry (row, k) = k·2^(off_row)·8B
//                  (+ 2^254·B on the top row), affine (y+x, y-x, 2dxy, -2dxy), row 0 holds ±2xy.
//   k_search<…>    one fused pass per key: seed (ChaCha20 / counter) -> SHA-512 -> clamp
//                  -> comb multiply from the table -> y as a fraction -> per-thread
//                  Montgomery batch + per-CTA pooled inversion -> canonical y -> base64
//                  values -> compare / shift-and / DFA match -> warp-ballot hit compaction.
//   k_derive<…>    full public keys (x too), an inversion per thread.
//
// Reference behaviour: src/service/gpu/kernel.cu:1898-2069 (meikey_search / meikey_derive).
// A launch covers the same consecutive indices from its base.
//
// Rates in comments are both sides of the change they explain, measured when it was made; later changes
// moved both.  As they stand the kernels run one needle at 0.95-0.98 G keys/s on hashed seeds and at
// 15.6 G on the incremental source (B200, long launches).
#include <cuda_runtime.h>
#include <stdint.h>

#include <algorithm>
#include <vector>

#include "ge.cuh"
#include "hash.cuh"
#include "kernels.h"

namespace mkb {

using mk32::fe;
using mk32::ge;
using mk32::niels;
using mk32::u32;
using mk32::u64;

// ---------------------------------------------------------------------------
// shared helpers
// ---------------------------------------------------------------------------

__device__ __forceinline__ fe load_fe(const uint4* p) {
    uint4 a = __ldg(p), b = __ldg(p + 1);
    fe r;
    r.v[0] = a.x; r.v[1] = a.y; r.v[2] = a.z; r.v[3] = a.w;
    r.v[4] = b.x; r.v[5] = b.y; r.v[6] = b.z; r.v[7] = b.w;
    return r;
}

__device__ __forceinline__ niels load_entry(const uint4* table, u64 idx) {
    const uint4* e = table + idx * (ENTRY_WORDS / 4);
    niels n;
    n.ypx = load_fe(e);
    n.ymx = load_fe(e + 2);
    n.t2d = load_fe(e + 4);
    return n;
}

// ---------------------------------------------------------------------------
// comb table build
// ---------------------------------------------------------------------------

__global__ void __launch_bounds__(256, 2) k_build_table(uint4* table, const CombGeom g, const u32* __restrict__ points,
                                                     u64 first, u64 count) {
    u64 e = first + (u64)blockIdx.x * blockDim.x + threadIdx.x;
    if (e >= first + count || e >= g.entries) return;
    u32 row = 0;
    for (u32 i = 1; i < g.rows; i++)
        if (e >= g.row_base[i]) row = i;
    u64 k = e - g.row_base[row];
    // points: per row R (X,Y,Z,T) then O (X,Y,Z,T), 8 words each; then 2d
    const u32* pr = points + (u64)row * 64;
    ge R, O;
    fe* rf[4] = {&R.X, &R.Y, &R.Z, &R.T};
    fe* of[4] = {&O.X, &O.Y, &O.Z, &O.T};
    for (int c = 0; c < 4; c++)
        for (int i = 0; i < 8; i++) {
            rf[c]->v[i] = pr[8 * c + i];
            of[c]->v[i] = pr[32 + 8 * c + i];
        }
    fe d2;
    for (int i = 0; i < 8; i++) d2.v[i] = points[(u64)g.rows * 64 + i];
    ge P = mk32::ge_identity();
    u32 nbits = 0;
    while (nbits < 63 && (g.cols[row] - 1) >> nbits) nbits++;
    for (int b = (int)nbits - 1; b >= 0; b--) {
        P = mk32::ge_add(P, P, d2);
        ge Q = mk32::ge_add(P, R, d2);
        if ((k >> b) & 1) P = Q;
    }
    P = mk32::ge_add(P, O, d2);
    fe zi = mk32::fe_invert(P.Z);
    fe x = mk32::fe_mul(P.X, zi), y = mk32::fe_mul(P.Y, zi);
    fe xy = mk32::fe_mul(x, y);
    fe t = row == 0 ? mk32::fe_add(xy, xy) : mk32::fe_mul(xy, d2);
    u32 w[32];
    mk32::fe_to_words(mk32::fe_add(y, x), w);
    mk32::fe_to_words(mk32::fe_sub(y, x), w + 8);
    mk32::fe_to_words(t, w + 16);
    mk32::fe_to_words(mk32::fe_sub(mk32::fe_zero(), t), w + 24);
    uint4* out = table + e * (COMB_STRIDE_WORDS / 4);
#pragma unroll
    for (int q = 0; q < 8; q++) out[q] = make_uint4(w[4 * q], w[4 * q + 1], w[4 * q + 2], w[4 * q + 3]);
}

// ---------------------------------------------------------------------------
// the fused key kernel
// ---------------------------------------------------------------------------

// Per-thread staging slots for the comb table: entry of row r is fetched with cp.async
// (16-byte LDGSTS, L2 only) into slot r & 1 one row ahead of its use.
struct EntrySlot {
    uint4 q[2][6];
};

// Fetches the entry of a signed digit as (y+x, y-x, 2dxy) of the digit's own point: a negative
// digit swaps the first two on their way into the slot and takes -2dxy, which the entry holds as
// its last 32 bytes, so the addition needs no selects (48 an addition).  With the tight sums of
// ge_add_niels and the rows of fe_mul that open a pair first, one addition takes 2320 instead of
// 2451 cycles of an SM sub-partition (16 warps per SM, the multiply pipe 93 % busy): hashed seeds
// 0.889 -> 0.926 G keys/s.
__device__ __forceinline__ void fetch_entry(EntrySlot& slot, int which, const uint4* table, u64 idx, bool neg) {
    const uint4* src = table + idx * (COMB_STRIDE_WORDS / 4);
    const u32 dst = (u32)__cvta_generic_to_shared(&slot.q[which][0]);
    const u32 lo = neg ? 32u : 0u;
    const uint4* t = src + (neg ? 6 : 4);
#pragma unroll
    for (int q = 0; q < 2; q++) {
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(dst + lo + 16 * q), "l"(src + q) : "memory");
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(dst + 32 - lo + 16 * q), "l"(src + 2 + q)
                     : "memory");
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(dst + 64 + 16 * q), "l"(t + q) : "memory");
    }
    asm volatile("cp.async.commit_group;\n" ::: "memory");
}

template <int N>
__device__ __forceinline__ void wait_entries() {
    asm volatile("cp.async.wait_group %0;\n" ::"n"(N) : "memory");
}

__device__ __forceinline__ niels read_entry(const EntrySlot& slot, int which) {
    niels n;
    const uint4* q = slot.q[which];
    uint4 a;
    a = q[0]; n.ypx.v[0] = a.x; n.ypx.v[1] = a.y; n.ypx.v[2] = a.z; n.ypx.v[3] = a.w;
    a = q[1]; n.ypx.v[4] = a.x; n.ypx.v[5] = a.y; n.ypx.v[6] = a.z; n.ypx.v[7] = a.w;
    a = q[2]; n.ymx.v[0] = a.x; n.ymx.v[1] = a.y; n.ymx.v[2] = a.z; n.ymx.v[3] = a.w;
    a = q[3]; n.ymx.v[4] = a.x; n.ymx.v[5] = a.y; n.ymx.v[6] = a.z; n.ymx.v[7] = a.w;
    a = q[4]; n.t2d.v[0] = a.x; n.t2d.v[1] = a.y; n.t2d.v[2] = a.z; n.t2d.v[3] = a.w;
    a = q[5]; n.t2d.v[4] = a.x; n.t2d.v[5] = a.y; n.t2d.v[6] = a.z; n.t2d.v[7] = a.w;
    return n;
}

// The digits of a clamped scalar's comb number m (bits 3..253 of s), lowest row first: m is
// shifted down by each row's width.
struct Digits {
    u32 m[8];
    int carry;
};

__device__ __forceinline__ Digits digits_of(const u64 s[4]) {
    Digits d;
    const u64 m[4] = {s[0] >> 3 | s[1] << 61, s[1] >> 3 | s[2] << 61, s[2] >> 3 | s[3] << 61,
                      (s[3] >> 3) & ((1ull << (251 - 192)) - 1ull)};
#pragma unroll
    for (int i = 0; i < 4; i++) {
        d.m[2 * i] = (u32)m[i];
        d.m[2 * i + 1] = (u32)(m[i] >> 32);
    }
    d.carry = 0;
    return d;
}

// the next row's digit; `top` (the last row): unsigned, the carry lands in it unchanged
__device__ __forceinline__ int next_digit(Digits& d, u32 w, bool top) {
    const int v = (int)(d.m[0] & ((1u << w) - 1u)) + d.carry;
#pragma unroll
    for (int i = 0; i < 7; i++) d.m[i] = __funnelshift_r(d.m[i], d.m[i + 1], w);
    d.m[7] >>= w;
    d.carry = top ? 0 : (v + (1 << (w - 1))) >> w;
    return v - (d.carry << w);
}

__device__ __forceinline__ u64 entry_index(const CombGeom& g, u32 row, int d) {
    return g.row_base[row] + (u64)(d < 0 ? -d : d);
}

// Row 0's entry in extended coordinates: X = 2x, Y = 2y, Z = 2, T = 2xy, without a multiplication
// (row 0 stores 2xy).
__device__ __forceinline__ ge comb_row0(const niels& n) {
    ge P;
    P.X = mk32::fe_tight(mk32::fe_sub_t(n.ypx, n.ymx));
    P.Y = mk32::fe_tight(mk32::fe_add_t(n.ypx, n.ymx));
    P.Z = mk32::fe_small(2);
    P.T = n.t2d;
    return P;
}

// Comb multiply: s (clamped, 4 LE words) -> y = yn/yd (and x = xn/xd when wanted).
// Row r's entry is fetched while row r-1 is being added.
__device__ __forceinline__ void comb_mul(const uint4* __restrict__ table, const CombGeom& g, const u64 s[4],
                                         EntrySlot& slot, fe& yn, fe& yd, fe* xn, fe* xd) {
    Digits dg = digits_of(s);
    const u32 rows = g.rows;
    auto fetch = [&](u32 row) {
        const int d = next_digit(dg, g.width[row], row + 1 == rows);
        fetch_entry(slot, row & 1, table, entry_index(g, row, d), d < 0);
    };
    fetch(0);
    fetch(1);
    wait_entries<1>();
    ge P = comb_row0(read_entry(slot, 0));
#pragma unroll 1
    for (u32 row = 1; row + 1 < rows; row++) {
        fetch(row + 1);
        wait_entries<1>();
        P = mk32::ge_add_niels(P, read_entry(slot, row & 1));
    }
    wait_entries<0>();
    mk32::ge_add_niels_frac(P, read_entry(slot, (rows - 1) & 1), yn, yd, xn, xd);
}

// 6-bit values of the 44-character base64 tail of the key blob (0x20 then the key),
// from the key's 8 little-endian words; only positions 1..43 are searched.
__device__ __forceinline__ u32 tail_value(const u32 pk[8], int pos) {
    // group g covers bytes b0 = (g ? pk[3g-1] : 0x20), pk[3g], pk[3g+1]
    int g = pos >> 2, k = pos & 3;
    auto byte = [&](int i) -> u32 { return (pk[i >> 2] >> (8 * (i & 3))) & 0xffu; };
    u32 b0 = g == 0 ? 32u : byte(3 * g - 1);
    u32 b1 = byte(3 * g);
    u32 b2 = 3 * g + 1 < 32 ? byte(3 * g + 1) : 0u;
    u32 n = b0 << 16 | b1 << 8 | b2;
    return (n >> (18 - 6 * k)) & 63u;
}

#define MK_SIGN_POS 42

// Walks the next N (or fewer) DFAs of the set `need` and takes them out of it, side by side so that
// their table lookups (shared memory when the launch staged the tables there, else global)
// overlap; sets the bits of those that may match.
template <int N>
__device__ __forceinline__ void dfa_walks(const MatchSet& ms, const u32 pk[8], u32& need, u64 hit_words[2]) {
    const uint16_t* t[N];
    u32 r[N], s[N], alt[N];
#pragma unroll
    for (int q = 0; q < N; q++) {
        r[q] = need ? (u32)__ffs((int)need) - 1u : r[0];
        need &= need - 1u;
        t[q] = reinterpret_cast<const uint16_t*>(ms.dfa[r[q]]);
        s[q] = alt[q] = 1;
    }
#pragma unroll 1
    for (int pos = 1; pos < 44; pos++) {
        const u32 v = tail_value(pk, pos);
#pragma unroll
        for (int q = 0; q < N; q++) {
            if (pos == MK_SIGN_POS) alt[q] = t[q][s[q] * 65u + (v | 2u)];
            else if (pos > MK_SIGN_POS) alt[q] = t[q][alt[q] * 65u + v];
            s[q] = t[q][s[q] * 65u + v];
        }
    }
#pragma unroll
    for (int q = 0; q < N; q++) {
        const bool ok = s[q] == 0 || t[q][s[q] * 65u + 64u] != 0 || alt[q] == 0 || t[q][alt[q] * 65u + 64u] != 0;
        const u32 id = ms.regex_id[r[q]];
        if (ok) hit_words[id >> 6] |= 1ull << (id & 63);
    }
}

// Whether some text needle of a quick-compare job (MatchSet::quick) may match the key: 3 operations a
// position instead of a table lookup and 6 (one needle on B200: 0.924 -> 0.929 G keys/s, incremental
// 11.5 -> 12.6, a suffix 13.2).  The bit of position 42 that the x sign decides is left
// out of every comparison.
__device__ __forceinline__ bool quick_match(const MatchSet& ms, const u32 pk[8]) {
    // the key as a big-endian bit string; character p starts at bit 6p - 8 (p = 1 with two zero bits
    // of the byte before the key)
    u32 k[9];
#pragma unroll
    for (int i = 0; i < 8; i++) k[i] = mkh::bswap32(pk[i]);
    k[8] = 0;
    bool any = false;
    for (u32 n = 0; n < ms.n_quick_contains; n++) {
        const u32 value = ms.quick_value[n], mask = ms.quick_mask[n];
#pragma unroll
        for (int p = 1; p <= 41; p++) {  // 3 characters fit at 41; a longer needle only passes too often
            const int bit = 6 * p - 8;
            const u32 w = p == 1 ? k[0] >> 2 : __funnelshift_l(k[bit / 32 + 1], k[bit / 32], bit % 32);
            const int sign = 248 - bit;  // the sign's place in the window
            const u32 m = sign < 32 ? mask & ~(0x80000000u >> (sign & 31)) : mask;
            any |= ((w ^ value) & m) == 0;
        }
    }
    for (u32 n = 0; n < ms.n_quick_suffix; n++)
        any |= ((k[7] ^ ms.quick_value[QUICK_CONTAINS + n]) & ms.quick_mask[QUICK_CONTAINS + n] & ~0x80u) == 0;
    return any;
}

// Tests one key (y only; the character at position 42 is tried with both x signs, as
// kernel.cu:1804-1875 does) and sets bit `id` of hit_words for every needle that may match.
// `lane_masks` and `lane_buckets` are tables with every value's entry once per lane, so that every lane
// reads its own banks: the low half of mask word 0 for jobs whose text needles fit in 32 bits of state
// (value v of lane l at v * 32 + l), and the bucket filter, whose 64-bit entries are read half a warp at a
// time (value v of lanes l and l + 16 at v * 16 + l).  Called by all 32 lanes of a warp.
// LIGHT: the job has neither the prefilter nor regex needles; their code costs the kernel
// registers (spills) that a job of a few needles runs faster without (one needle on B200: 0.929 ->
// 0.936 G keys/s, incremental 12.6 -> 12.9).
template <bool LIGHT>
__device__ __forceinline__ void match_key(const MatchSet& ms, const u32* lane_masks, const u64* lane_buckets,
                                          const u32 pk[8], u64 hit_words[2]) {
    hit_words[0] = hit_words[1] = 0;
    u32 words = ms.sa_words;
    if (ms.quick && !quick_match(ms, pk)) {
        if (LIGHT || ms.n_regex == 0) return;
        words = 0;
    }
    auto value = [&](int pos) { return tail_value(pk, pos); };  // cut out where used: 43 of them do not stay in registers
    // text needles: shift-and over sa_words words of state.  With the 4-gram prefilter, the
    // words of the needles of 4+ characters are scanned only when one of the key's 4-character
    // windows (position 42 with both values) is the start of such a needle.  The bitmap's lookups
    // are a cache line per lane, 32 a load, and bound the L1 tag stage (5200 of 46700 cycles a key
    // for 58 needles on B200), so the bucket filter in shared memory lets about one key in a hundred
    // through to them (58 needles; half of them at 128).
    u32 flags = ~0u;  // the buckets the key may hold something of
    if (!LIGHT && ms.buckets) {
        const u64* lm = lane_buckets + (threadIdx.x & 15u);
        u64 D = 0;
        u32 acc = 0;
#pragma unroll
        for (int pos = 1; pos < 44; pos++) {
            u64 mk = lm[value(pos) * 16u];
            if (pos == MK_SIGN_POS) mk |= lm[(value(pos) | 2u) * 16u];
            D = (D << BUCKETS | ((1ull << BUCKETS) - 1)) & mk;
            acc |= (u32)(D >> 32);
        }
        D = D << BUCKETS & ms.bucket_end;
        acc |= (u32)((D | (D << BUCKETS & ms.bucket_end)) >> 32);
        flags = acc >> (BUCKETS * (BUCKET_CHARS - 1) - 32);
    }
    if (!LIGHT && ms.gram4) {
        u32 any = 0;
        if (flags & ms.text_buckets) {
            u32 gw = value(1) << 12 | value(2) << 6 | value(3);
#pragma unroll
            for (int p = 1; p + 3 < 44; p++) {
                gw = (gw << 6 | value(p + 3)) & 0xffffffu;
                any |= __ldg(ms.gram4 + (gw >> 5)) >> (gw & 31);
                if (p <= MK_SIGN_POS && MK_SIGN_POS <= p + 3) {
                    const u32 g2 = gw | 2u << (6 * (p + 3 - MK_SIGN_POS));
                    any |= __ldg(ms.gram4 + (g2 >> 5)) >> (g2 & 31);
                }
            }
        }
        if (!(any & 1u)) words = ms.short_words;
    }
    u32 scanned = 0;
    if (ms.narrow && words) {
        const u32* lm = lane_masks + (threadIdx.x & 31u);
        u32 D = 0, acc = 0;
        const u32 first = (u32)ms.first_bit[0], last = (u32)ms.last_bit[0];
#pragma unroll
        for (int pos = 1; pos < 44; pos++) {
            u32 mk = lm[value(pos) * 32u];
            if (pos == MK_SIGN_POS) mk |= lm[(value(pos) | 2u) * 32u];
            D = ((D << 1) | first) & mk;
            acc |= D & last;
        }
        acc |= D & (u32)ms.suffix_bit[0];
        for (u32 t = 0; acc && t < ms.n_text; t++) {
            const u32 b = ms.text_last[t];
            if (b < 32u && ((acc >> b) & 1u)) {
                const u32 id = ms.text_id[t];
                hit_words[id >> 6] |= 1ull << (id & 63);
            }
        }
        scanned = 1;
    }
    for (u32 wi = scanned; wi < words; wi++) {
        u64 D = 0, acc = 0;
        u64 first = ms.first_bit[wi], last = ms.last_bit[wi];
#pragma unroll
        for (int pos = 1; pos < 44; pos++) {
            u64 mk = ms.mask[wi][value(pos)];
            if (pos == MK_SIGN_POS) mk |= ms.mask[wi][value(pos) | 2u];
            D = ((D << 1) | first) & mk;
            acc |= D & last;
        }
        acc |= D & ms.suffix_bit[wi];
        if (acc) {
            // map bits to needles
            for (u32 t = 0; t < ms.n_text; t++) {
                u32 b = ms.text_last[t];
                if ((b >> 6) == wi && ((acc >> (b & 63)) & 1)) {
                    u32 id = ms.text_id[t];
                    hit_words[id >> 6] |= 1ull << (id & 63);
                }
            }
        }
    }
    // regex needles: the walks of those that the warp's keys cannot be told from by the buckets (8 DFAs
    // of the multi-pattern workload on B200: 5 have buckets and are walked by every seventh warp, 0.850 ->
    // 0.865 G keys/s alone and 0.807 -> 0.818 beside 64 text needles)
    if (!LIGHT && ms.n_regex) {
        u32 need = ms.regex_always;
        for (u32 i = 0; i < ms.n_filtered; i++) need |= ((flags >> (BUCKETS - 1 - i)) & 1u) << ms.filtered[i];
        need = __reduce_or_sync(0xffffffffu, need);
        while (need)
            if (__popc(need) > 4) dfa_walks<8>(ms, pk, need, hit_words);
            else dfa_walks<4>(ms, pk, need, hit_words);
    }
}

// Warp-compacted hit output: lanes with hits take consecutive ring slots with one
// atomicAdd per warp (inclusive scan of the per-lane hit counts).  Called by all 32 lanes.
__device__ __forceinline__ void report_hits(const u64 hw[2], u64 index, HitRecord* hits, u32 cap, JobDevice* jd) {
    const u32 lane = threadIdx.x & 31u;
    u32 cnt = (u32)(__popcll(hw[0]) + __popcll(hw[1]));
    u32 incl = cnt;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        u32 y = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= (u32)o) incl += y;
    }
    u32 total = __shfl_sync(0xffffffffu, incl, 31);
    u32 base = 0;
    if (lane == 31) base = atomicAdd(&jd->hit_count, total);
    base = __shfl_sync(0xffffffffu, base, 31);
    u32 slot = base + incl - cnt;
    for (int w = 0; w < 2; w++) {
        u64 bits = hw[w];
        while (bits) {
            int b = __ffsll((long long)bits) - 1;
            bits &= bits - 1;
            if (slot < cap) {
                hits[slot].index = index;
                hits[slot].needle = (u32)(w * 64 + b);
                hits[slot].reserved = 0;
            }
            slot++;
        }
    }
}

// Seed of index `idx` -> clamped scalar.  `blk`/`blk_id` cache the ChaCha20 block
// shared by an even index and the next odd one.
__device__ __forceinline__ void scalar_of(u32 seed_src, const u32 key[8], const mkh::CounterMid& mid, u64 idx,
                                          u32 blk[16], u64& blk_id, u64 s[4]) {
    if (seed_src == 1) {
        mkh::counter_scalar(mid, idx, s);
    } else {
        if ((idx >> 1) != blk_id) {
            blk_id = idx >> 1;
            mkh::chacha20_block(key, blk_id, blk);
        }
        u32 sw[8];
        const bool odd = idx & 1;
#pragma unroll
        for (int i = 0; i < 8; i++) sw[i] = odd ? blk[8 + i] : blk[i];
        mkh::seed_scalar(sw, s);
    }
}

// Batch state of one iteration of one thread (Montgomery's trick with two field elements
// per key): a[j] = num_j · den_0 ··· den_(j-1) and den[j]; `prod` = den_0 ··· den_(KPT-1).
// With inv = 1/prod the back-sweep gives y_j = a[j] · inv_j, inv_(j-1) = inv_j · den[j].
template <int KPT>
struct Batch {
    fe a[KPT], den[KPT];
    fe prod;
};

// Seeds and clamped scalars of KPT consecutive indices (ALU work: ChaCha20, SHA-512).
template <int KPT>
__device__ __forceinline__ void scalars(const KeyLaunch& L, const u32 key[8], const mkh::CounterMid& mid, u64 first,
                                        u64 sc[KPT][4]) {
    u32 blk[16];
    u64 blk_id = ~0ull;
#pragma unroll 1
    for (int j = 0; j < KPT; j++) scalar_of(L.seed_src, key, mid, first + (u64)j, blk, blk_id, sc[j]);
}

__device__ __forceinline__ niels smem_niels(const uint4* q);

// Comb multiply with the whole table in shared memory (entries 96 bytes apart, `stab`): every
// row reads its entry there, with no staging; y = yn/yd only.
__device__ __forceinline__ void comb_mul_smem(const uint4* stab, const CombGeom& g, const u64 s[4], fe& yn, fe& yd) {
    Digits dg = digits_of(s);
    const u32 rows = g.rows;
    auto entry = [&](u32 row) {
        const int d = next_digit(dg, g.width[row], row + 1 == rows);
        return mk32::niels_signed(smem_niels(stab + entry_index(g, row, d) * 6), d < 0);
    };
    ge P = comb_row0(entry(0));
#pragma unroll 1
    for (u32 row = 1; row + 1 < rows; row++) P = mk32::ge_add_niels(P, entry(row));
    mk32::ge_add_niels_frac(P, entry(rows - 1), yn, yd, nullptr, nullptr);
}

// Comb multiplies of the KPT scalars (IMAD work) into the batch; STAB: from the table in
// shared memory.
template <int KPT, bool STAB = false>
__device__ __forceinline__ void combs(const KeyLaunch& L, const CombGeom& g, const u64 sc[KPT][4], EntrySlot& slot,
                                      const uint4* stab, Batch<KPT>& b) {
    fe run;
#pragma unroll 1
    for (int j = 0; j < KPT; j++) {
        fe num;
        if (STAB) comb_mul_smem(stab, g, sc[j], num, b.den[j]);
        else comb_mul(L.table, g, sc[j], slot, num, b.den[j], nullptr, nullptr);
        if (j == 0) {
            b.a[0] = num;
            run = b.den[0];
        } else {
            b.a[j] = mk32::fe_mul(num, run);
            run = mk32::fe_mul(run, b.den[j]);
        }
    }
    b.prod = run;
}

// The key (0 .. KPT-1) in slot s of an incremental batch.
template <int KPT>
__device__ __forceinline__ int incr_key(int s) {
    const int d = (s + 1) >> 1;
    return s == KPT - 1 ? 0 : (s & 1) ? KPT / 2 + d : KPT / 2 - d;
}

// Backward pass: `inv` is 1/(product of the batch's denominators); yields each key's
// canonical y (sign bit 0), tests the needles and reports candidate hits (none when `valid` is
// false: a run past the launch's last one).  INCR: slot j holds key incr_key(j).
template <int KPT, bool INCR, bool LIGHT>
__device__ __forceinline__ void backward(const KeyLaunch& L, const MatchSet& ms, const u32* lane_masks,
                                         const u64* lane_buckets, u64 first, bool valid, const Batch<KPT>& b, fe inv,
                                         u32& sink) {
    // a key's two elements are loaded while the one before is tested (they have gone to the L2 cache
    // and further since the forward pass): on B200 incremental 13.0 -> 14.5, hashed 0.974 -> 0.980 G keys/s
    fe a = b.a[KPT - 1], den = b.den[KPT - 1];
#pragma unroll 1
    for (int j = KPT - 1; j >= 0; j--) {
        const int next = j > 0 ? j - 1 : 0;
        const fe a_next = b.a[next], den_next = b.den[next];
        u32 pk[8];
        mk32::fe_to_words(mk32::fe_mul(a, inv), pk);
        if (j > 0) inv = mk32::fe_mul(inv, den);
        a = a_next;
        den = den_next;
        sink ^= pk[7];
        u64 hw[2];
        match_key<LIGHT>(ms, lane_masks, lane_buckets, pk, hw);
        if (!valid) hw[0] = hw[1] = 0;
        const bool any = (hw[0] | hw[1]) != 0;
        // warp ballot: the (rare) warps with a hit compact their records into the ring
        if (__ballot_sync(0xffffffffu, any)) report_hits(hw, first + (u64)(INCR ? incr_key<KPT>(j) : j), L.hits, L.hit_cap, L.job);
    }
}

// Named barriers of the search pipeline: products of buffer b ready (1 + b), inverses of
// buffer b ready (3 + b).  Barrier 0 is __syncthreads.
__device__ __forceinline__ void bar_sync(int id, int count) { asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(count) : "memory"); }
__device__ __forceinline__ void bar_arrive(int id, int count) { asm volatile("bar.arrive %0, %1;" ::"r"(id), "r"(count) : "memory"); }

// Inverts the n products prod[0 .. n) in place with one field inversion per pool: lane l < pools
// of the calling warp handles the strided pool l, l+pools, l+2·pools, ... (Montgomery's trick
// inside each pool); the other lanes idle.  With 32 pools every lane works; fewer pools share
// each inversion among more keys (the inversion batch of a pool is its products x the keys per
// thread).
__device__ __forceinline__ void invert_pools(fe* prod, fe* scratch, int n, int pools = 32) {
    const int l = threadIdx.x & 31;
    if (l >= pools) return;
    const int groups = (n - l + pools - 1) / pools;
    fe acc = prod[l];
    scratch[l] = acc;
#pragma unroll 1
    for (int k = 1; k < groups; k++) {
        acc = mk32::fe_mul(acc, prod[l + pools * k]);
        scratch[l + pools * k] = acc;
    }
    fe inv = mk32::fe_invert(acc);
#pragma unroll 1
    for (int k = groups - 1; k > 0; k--) {
        fe t = mk32::fe_mul(inv, scratch[l + pools * (k - 1)]);
        inv = mk32::fe_mul(inv, prod[l + pools * k]);
        prod[l + pools * k] = t;
    }
    prod[l] = inv;
}

// ---------------------------------------------------------------------------
// incremental source: index base + i is the point (s0 + base + i)·B
// ---------------------------------------------------------------------------

__device__ __forceinline__ fe words_fe(const u32* w) {
    fe r;
#pragma unroll
    for (int i = 0; i < 8; i++) r.v[i] = w[i];
    return r;
}

__device__ __forceinline__ niels words_niels(const u32* w) {
    niels n;
    n.ypx = words_fe(w);
    n.ymx = words_fe(w + 8);
    n.t2d = words_fe(w + 16);
    return n;
}

__device__ __forceinline__ niels smem_niels(const uint4* q) {
    niels n;
    uint4 a;
    a = q[0]; n.ypx.v[0] = a.x; n.ypx.v[1] = a.y; n.ypx.v[2] = a.z; n.ypx.v[3] = a.w;
    a = q[1]; n.ypx.v[4] = a.x; n.ypx.v[5] = a.y; n.ypx.v[6] = a.z; n.ypx.v[7] = a.w;
    a = q[2]; n.ymx.v[0] = a.x; n.ymx.v[1] = a.y; n.ymx.v[2] = a.z; n.ymx.v[3] = a.w;
    a = q[3]; n.ymx.v[4] = a.x; n.ymx.v[5] = a.y; n.ymx.v[6] = a.z; n.ymx.v[7] = a.w;
    a = q[4]; n.t2d.v[0] = a.x; n.t2d.v[1] = a.y; n.t2d.v[2] = a.z; n.t2d.v[3] = a.w;
    a = q[5]; n.t2d.v[4] = a.x; n.t2d.v[5] = a.y; n.t2d.v[6] = a.z; n.t2d.v[7] = a.w;
    return n;
}

// The launch's start point (s0 + base)·B plus offset·B from the 4-bit window table
// (offset < 2^32; one mixed addition per nonzero window).
__device__ __forceinline__ ge incr_start(const KeyLaunch& L, u64 offset) {
    ge P;
    P.X = words_fe(L.start);
    P.Y = words_fe(L.start + 8);
    P.Z = words_fe(L.start + 16);
    P.T = words_fe(L.start + 24);
#pragma unroll 1
    for (int w = 0; w < INCR_WINDOWS; w++) {
        const u32 d = (u32)(offset >> (4 * w)) & 15u;
        if (d) P = mk32::ge_add_niels(P, load_entry(L.incr, (u64)w * 16 + d));
    }
    return P;
}

// Copies the step table j·B (j = 0 .. INCR_STEPS-1) into shared memory.
__device__ __forceinline__ void load_steps(const KeyLaunch& L, uint4* steps, u32 tid, u32 nthr) {
    const uint4* src = L.incr + (u64)INCR_WINDOWS * 16 * (ENTRY_WORDS / 4);
    for (u32 i = tid; i < (u32)INCR_STEPS * (ENTRY_WORDS / 4); i += nthr) steps[i] = src[i];
}

// Turns entry j of a copied step table from (y+x, y-x, 2dxy) into (2y, 2x, 2dxy).
__device__ __forceinline__ void step_to_yx(uint4* steps, u32 j) {
    uint4* e = steps + j * (ENTRY_WORDS / 4);
    const niels n = smem_niels(e);
    const fe y = mk32::fe_add(n.ypx, n.ymx), x = mk32::fe_sub(n.ypx, n.ymx);
    e[0] = make_uint4(y.v[0], y.v[1], y.v[2], y.v[3]);
    e[1] = make_uint4(y.v[4], y.v[5], y.v[6], y.v[7]);
    e[2] = make_uint4(x.v[0], x.v[1], x.v[2], x.v[3]);
    e[3] = make_uint4(x.v[4], x.v[5], x.v[6], x.v[7]);
}

// Batch of the KPT consecutive points around Q: Q + (j - KPT/2)·B for j = 0 .. KPT-1.  Q and
// the points Q ± d·B share their products: with a step's (2y, 2x, 2dxy),
//   y(Q ± dB) = (Y·2y ± X·2x) / (2Z -+ T·2dxy),
// three multiplications for two keys instead of three for each.  On B200, 2^30 candidates at 16
// keys per thread: 96.5 ms, against 109.0 ms with one mixed addition per key.
// The batch's slots are filled in the order Q, +1, -1, +2, -2, ..., -KPT/2 (incr_key).
template <int KPT>
__device__ __forceinline__ void incr_fracs(const ge& Q, const uint4* steps, Batch<KPT>& b) {
    const fe z2 = mk32::fe_add_t(Q.Z, Q.Z);
    b.a[0] = Q.Y;
    b.den[0] = Q.Z;
    fe run = Q.Z;
#pragma unroll 1
    for (int d = 1; d <= KPT / 2; d++) {
        const niels t = smem_niels(steps + d * (ENTRY_WORDS / 4));  // (2y, 2x, 2dxy)
        const fe yy = mk32::fe_mul(Q.Y, t.ypx), xx = mk32::fe_mul(Q.X, t.ymx), c = mk32::fe_mul(Q.T, t.t2d);
        if (d < KPT / 2) {
            const fe den = mk32::fe_sub_t(z2, c);
            b.den[2 * d - 1] = den;
            b.a[2 * d - 1] = mk32::fe_mul(mk32::fe_add_t(yy, xx), run);
            run = mk32::fe_mul(run, den);
        }
        const int s = d < KPT / 2 ? 2 * d : KPT - 1;
        const fe den = mk32::fe_add_1(z2, c);
        b.den[s] = den;
        b.a[s] = mk32::fe_mul(mk32::fe_sub_t(yy, xx), run);
        run = mk32::fe_mul(run, den);
    }
    b.prod = run;
}

// Search kernel.  The launch's keys are L.chunks runs of KPT consecutive indices.  Each compute
// thread takes one run per iteration: warp w of CTA c takes runs ((it·warps + w)·CTAs + c)·32 + lane,
// so a last iteration with fewer runs than threads leaves whole warps out, spread over the SMs
// (they only take part in the barriers).  Iterations are pipelined two deep: a compute thread runs
// the forward pass of iteration it before the backward pass of it-1, and the CTA's products of an
// iteration are turned into their inverses in between.  Who inverts:
//   ROT true (hashed seeds): every warp computes keys, and the inversion of iteration it falls to
//     warp it mod the CTA's warps, so that consecutive inversions run on different SM
//     sub-partitions and every warp carries the same share.  A dedicated inverter leaves its
//     sub-partition with three compute warps against four (warp w runs on sub-partition w % 4):
//     on B200, 8 keys per thread, 0.82 -> 0.89 G keys/s with the rotating duty.  The inverting
//     warp does its backward pass of it-1 first: by then the others have arrived, so it does not
//     wait for the slowest of them, and they still have a whole forward pass to run before they need
//     the inverses (0.936 -> 0.974 G keys/s; 0.916 -> 0.966 at 16 pools, whose chain is longer);
//   ROT false (the incremental source, whose iterations are an order shorter): the CTA's last warp,
//     which does nothing else (BLOCK-32 compute threads), so the inversion's dependent chain runs
//     beside the other warps' work (11.0 against 8.8 G keys/s with the rotating duty).
// The CTA's CT products of an iteration are inverted in L.inv_pools pools (default 32: lane l
// of the inverting warp takes threads l, l+32, ...), one field inversion each, so one
// inversion serves about KPT·CT/pools keys.
// Hashed seeds run 8 keys per thread whatever the context's keys per thread (which sets the
// launch's span): 4 keys share the barriers among too few (0.78 against 0.895 G keys/s), and 16
// gain 0.3 % on long launches only (0.983 against 0.980) while a launch of one or two iterations has
// less to overlap.
// The incremental source runs 16: its step point and inversion are shared by the batch (7.0 G keys/s
// at 4, 10.7 at 8, 14.5 at 16).
// The one call of the forward pass stands inside the loop: a second one for the first iteration
// makes the compiler keep it out of line, with the batch behind pointers (0.83 against 0.895 G
// keys/s).
// Named barriers, all BLOCK threads: products of buffer b ready (1 + b): the inverting warp
// waits, the others arrive; inverses of buffer b ready (3 + b): the inverting warp arrives,
// the others wait.  Stop requests (host stop word, or a hit with stop_on_hit) are read by
// the inverting warp and take effect two iterations later, at a point every warp agrees on
// (tests/test_search_buffers.py model-checks both forms with their accesses to the buffers).
// INCR: the incremental source.  A compute thread keeps the point Q of its middle index (key
// KPT/2) in the current iteration; its keys are Q ± d·B from the step table, and Q advances by
// CTAs·CT·KPT·B (one mixed addition) per iteration.  No comb table is read.
// STAB: the comb table lives in shared memory (copied by every CTA at the start, in place of
// the staging slots; tables of a few hundred to a few thousand entries, 40+ rows).
template <int KPT, int BLOCK, bool INCR, bool ROT, bool LIGHT, bool STAB = false>
__global__ void __launch_bounds__(BLOCK, 512 / BLOCK) k_search(const KeyLaunch L) {
    constexpr int CT = ROT ? BLOCK : BLOCK - 32;  // compute threads
    constexpr int CW = CT / 32;                   // compute warps
    extern __shared__ uint4 dyn_smem[];
    fe (*prod)[CT] = reinterpret_cast<fe (*)[CT]>(dyn_smem);
    fe* scratch = prod[2];  // one inversion runs at a time: the next one waits for this one's warp
    EntrySlot* slots = reinterpret_cast<EntrySlot*>(scratch + CT);
    uint4* stab = reinterpret_cast<uint4*>(scratch + CT);  // STAB: the table in place of the slots
    __shared__ CombGeom g;
    __shared__ MatchSet ms;
    __shared__ u32 lane_masks[64 * 32];  // see match_key
    __shared__ u64 lane_buckets[LIGHT ? 1 : 64 * 16];
    __shared__ u32 key[8];
    __shared__ mkh::CounterMid mid;
    __shared__ volatile u64 stop_iter;
    __shared__ uint4 steps[INCR ? INCR_STEPS * (ENTRY_WORDS / 4) : 1];
    const u32 tid = threadIdx.x;
    const u64 nthreads = (u64)gridDim.x * CT;
    const u64 iters = (L.chunks + nthreads - 1) / nthreads;
    if (INCR) load_steps(L, steps, tid, BLOCK);
    {
        const u32* src = (const u32*)&L.geom;
        u32* dst = (u32*)&g;
        for (u32 i = tid; i < sizeof(CombGeom) / 4; i += BLOCK) dst[i] = src[i];
        const u32* s2 = (const u32*)L.match;
        u32* d2 = (u32*)&ms;
        for (u32 i = tid; i < sizeof(MatchSet) / 4; i += BLOCK) d2[i] = s2[i];
        if (tid < 8) key[tid] = L.key[tid];
        if (tid == 0) stop_iter = iters;
    }
    __syncthreads();
    if (STAB)  // entries 128 bytes apart in HBM, 96 here
        for (u32 e = tid; e < (u32)g.entries; e += BLOCK)
#pragma unroll
            for (int q = 0; q < 6; q++) stab[e * 6 + q] = L.table[(u64)e * (COMB_STRIDE_WORDS / 4) + q];
    if (!LIGHT && L.dfa_smem) {
        // stage the job's DFA tables behind the other dynamic buffers, those that every key walks first,
        // as many as the launch reserved room for, and point the matcher at the copies (16-byte aligned
        // tables, copied in u16 units)
        uint8_t* area = reinterpret_cast<uint8_t*>(INCR ? (void*)slots : (void*)(slots + CT));
        auto each_staged = [&](auto f) {
            u32 off = 0;
            for (u32 rest = 0; rest < 2; rest++)
                for (u32 r = 0; r < ms.n_regex; r++) {
                    const u32 bytes = (ms.dfa_states[r] * 130u + 15u) & ~15u;
                    if (((ms.regex_always >> r) & 1u) == rest || bytes > L.dfa_smem - off) continue;
                    f(r, area + off);
                    off += bytes;
                }
        };
        each_staged([&](u32 r, uint8_t* to) {
            const uint16_t* src = reinterpret_cast<const uint16_t*>(ms.dfa[r]);
            uint16_t* dst = reinterpret_cast<uint16_t*>(to);
            for (u32 i = tid; i < ms.dfa_states[r] * 65u; i += BLOCK) dst[i] = src[i];
        });
        __syncthreads();
        if (tid == 0) each_staged([&](u32 r, uint8_t* to) { ms.dfa[r] = to; });
    }
    if (ms.narrow)
        for (u32 i = tid; i < 64u * 32u; i += BLOCK) lane_masks[i] = (u32)ms.mask[0][i >> 5];
    if (!LIGHT && ms.buckets)
        for (u32 i = tid; i < 64u * 16u; i += BLOCK) lane_buckets[i] = ms.bucket[i >> 4];
    if (INCR && tid < (u32)INCR_STEPS) step_to_yx(steps, tid);
    if (tid == 0 && L.seed_src == 1) mid = mkh::counter_mid(key);
    __syncthreads();
    if (iters == 0) return;
    const int pools = (int)L.inv_pools;  // inversion pools of the CTA, 1..32
    auto read_stop = [&](u64 it) {       // by the inverting warp
        if ((tid & 31) == 0) {
            const volatile JobDevice* jd = L.job;
            if ((jd->stop != 0 || (L.stop_on_hit && jd->hit_count != 0)) && it + 2 < stop_iter) stop_iter = it + 2;
        }
        __syncwarp();
    };

    if (!ROT && tid >= (u32)CT) {
        // ---- dedicated inverter warp ----
        for (u64 it = 0;; it++) {
            const int b = it & 1;
            bar_sync(1 + b, BLOCK);
            read_stop(it);
            invert_pools(prod[b], scratch, CT, pools);
            __syncwarp();
            bar_arrive(3 + b, BLOCK);
            if (it + 1 >= iters || it + 1 >= stop_iter) break;
        }
        if ((tid & 31) == 0 && stop_iter < iters) atomicOr(&L.job->status, 1u);
        return;
    }

    // ---- compute warps ----
    const u32 warp = tid >> 5;
    auto inverts = [&](u64 it) { return ROT && warp == (u32)it % (u32)CW; };
    auto chunk_of = [&](u64 it) { return ((it * CW + warp) * gridDim.x + blockIdx.x) * 32u + (tid & 31u); };
    auto first_of = [&](u64 it) { return L.base + chunk_of(it) * KPT; };
    EntrySlot& slot = slots[INCR || STAB ? 0 : tid];
    Batch<KPT> batch[2];
    u64 sc[KPT][4];
    u32 sink = 0;
    ge Q;
    if (INCR) Q = incr_start(L, chunk_of(0) * KPT + KPT / 2);
    for (u64 it = 0;; it++) {
        if (it == 0 || (it < iters && it < stop_iter)) {
            // forward pass of iteration it
            const int b = it & 1;
            if (chunk_of(it) - (tid & 31u) >= L.chunks) {
                batch[b].prod = mk32::fe_small(1);  // a warp past the last run
            } else if (INCR) {
                incr_fracs<KPT>(Q, steps, batch[b]);
                Q = mk32::ge_add_niels(Q, words_niels(L.delta));
            } else {
                scalars<KPT>(L, key, mid, first_of(it), sc);
                combs<KPT, STAB>(L, g, sc, slot, stab, batch[b]);
            }
            prod[b][tid] = batch[b].prod;
            if (!inverts(it)) bar_arrive(1 + b, BLOCK);
        }
        if (it > 0) {
            // backward pass of iteration it - 1
            const u64 p = it - 1;
            const int b = p & 1;
            if (!inverts(p)) bar_sync(3 + b, BLOCK);
            if (chunk_of(p) - (tid & 31u) < L.chunks)
                backward<KPT, INCR, LIGHT>(L, ms, lane_masks, lane_buckets, first_of(p), chunk_of(p) < L.chunks, batch[b],
                                           prod[b][tid], sink);
            if (it >= iters || it >= stop_iter) break;
        }
        if (inverts(it)) {
            // iteration it was run: the loop ends above otherwise
            const int b = it & 1;
            bar_sync(1 + b, BLOCK);
            read_stop(it);
            invert_pools(prod[b], scratch, CT, pools);
            __syncwarp();
            bar_arrive(3 + b, BLOCK);
        }
    }
    // the decision of the iteration that ended the loop is visible here (its inverses were waited for)
    if (ROT && tid == 0 && stop_iter < iters) atomicOr(&L.job->status, 1u);
    if (L.sink) L.sink[(u64)blockIdx.x * CT + tid] = sink;
}

constexpr int DERIVE_BLOCK = 128;

// Derive kernel: full public keys (x sign included) of indices base .. base+count-1, KPT
// consecutive ones per thread, with one inversion of its 2·KPT denominators per thread.  INCR: the
// thread's keys are Q + j·B with Q = (s0 + first)·B; key j gives y = (b+a)/(2Z-c) and
// x = (b-a)/(2Z+c) of the mixed addition with step entry j (entry 0 is the identity).
// Threads do not work together: with the division steps an inversion costs about two thirds of a
// key, and a call of few keys is a single dependent chain per thread, so the keys go to as many
// threads as one wave holds (launch_derive) instead of waiting behind each other.
template <int KPT, bool INCR>
__global__ void __launch_bounds__(DERIVE_BLOCK, 512 / DERIVE_BLOCK) k_derive(const KeyLaunch L) {
    constexpr int NUM = 2 * KPT;
    extern __shared__ uint4 dyn_smem[];
    EntrySlot* slots = reinterpret_cast<EntrySlot*>(dyn_smem);
    __shared__ CombGeom g;
    __shared__ u32 key[8];
    __shared__ uint4 steps[INCR ? INCR_STEPS * (ENTRY_WORDS / 4) : 1];
    const u32 tid = threadIdx.x;
    const u64 gid = (u64)blockIdx.x * DERIVE_BLOCK + tid;
    if (INCR) load_steps(L, steps, tid, DERIVE_BLOCK);
    {
        const u32* src = (const u32*)&L.geom;
        u32* dst = (u32*)&g;
        for (u32 i = tid; i < sizeof(CombGeom) / 4; i += DERIVE_BLOCK) dst[i] = src[i];
        if (tid < 8) key[tid] = L.key[tid];
    }
    __syncthreads();
    if (gid * KPT >= L.count) return;
    mkh::CounterMid mid;
    if (L.seed_src == 1) mid = mkh::counter_mid(key);
    const u64 first = L.base + gid * KPT;
    fe num[NUM], den[NUM], pre[NUM];
    u32 blk[16];
    u64 blk_id = ~0ull;
    ge Q;
    fe ypx, ymx, z2;
    if (INCR) {
        Q = incr_start(L, gid * KPT);
        ypx = mk32::fe_add_t(Q.Y, Q.X);
        ymx = mk32::fe_sub_t(Q.Y, Q.X);
        z2 = mk32::fe_add_t(Q.Z, Q.Z);
    }
#pragma unroll 1
    for (int j = 0; j < KPT; j++) {
        if (INCR) {
            const niels t = smem_niels(steps + j * (ENTRY_WORDS / 4));
            const fe A = mk32::fe_mul(ymx, t.ymx), B = mk32::fe_mul(ypx, t.ypx), C = mk32::fe_mul(Q.T, t.t2d);
            num[2 * j] = mk32::fe_add_t(B, A);
            den[2 * j] = mk32::fe_sub_t(z2, C);
            num[2 * j + 1] = mk32::fe_sub_t(B, A);
            den[2 * j + 1] = mk32::fe_add_1(z2, C);
        } else {
            u64 s[4];
            scalar_of(L.seed_src, key, mid, first + (u64)j, blk, blk_id, s);
            comb_mul(L.table, g, s, slots[tid], num[2 * j], den[2 * j], &num[2 * j + 1], &den[2 * j + 1]);
        }
        pre[2 * j] = j == 0 ? den[0] : mk32::fe_mul(pre[2 * j - 1], den[2 * j]);
        pre[2 * j + 1] = mk32::fe_mul(pre[2 * j], den[2 * j + 1]);
    }
    fe inv = mk32::fe_invert(pre[NUM - 1]);
#pragma unroll 1
    for (int j = KPT - 1; j >= 0; j--) {
        const u64 at = gid * KPT + (u64)j;
        const int ex = 2 * j + 1, ey = 2 * j;
        fe xinv = mk32::fe_mul(inv, pre[ex - 1]);
        inv = mk32::fe_mul(inv, den[ex]);
        fe yinv = ey == 0 ? inv : mk32::fe_mul(inv, pre[ey - 1]);
        if (ey > 0) inv = mk32::fe_mul(inv, den[ey]);
        u32 xw[8], pk[8];
        mk32::fe_to_words(mk32::fe_mul(num[ex], xinv), xw);
        mk32::fe_to_words(mk32::fe_mul(num[ey], yinv), pk);
        pk[7] |= (xw[0] & 1u) << 31;
        if (at < L.count) {
            uint4* o = (uint4*)(L.out + at * 32);
            o[0] = make_uint4(pk[0], pk[1], pk[2], pk[3]);
            o[1] = make_uint4(pk[4], pk[5], pk[6], pk[7]);
        }
    }
}

// ---------------------------------------------------------------------------
// host launch wrappers
// ---------------------------------------------------------------------------

// dynamic shared memory of a search: products (two buffers), inversion scratch and the
// per-thread table staging slots (the incremental source reads no comb table and needs none)
static size_t dyn_bytes(bool incr, uint32_t block, uint32_t table_smem) {
    const size_t fe_bytes = 32, threads = search_kernel_threads(incr, block, table_smem);
    if (table_smem && !incr) return 3 * threads * fe_bytes + table_smem;  // the table in place of the slots
    return 3 * threads * fe_bytes + (incr ? 0 : threads * sizeof(EntrySlot));
}

// search kernels with the comb table in shared memory: the dedicated-inverter layout, block
// 512, keys per thread 4 and 8
static const void* stab_kernel_of(uint32_t kpt, uint32_t block) {
    if (block != 512) return nullptr;
    if (kpt == 4) return (const void*)k_search<4, 512, false, false, false, true>;
    if (kpt == 8) return (const void*)k_search<8, 512, false, false, false, true>;
    return nullptr;
}

template <bool LIGHT>
static const void* kernel_of(bool incr, uint32_t block) {
#define MK_FN(B) \
    if (block == B) \
        return incr ? (const void*)k_search<INCR_KEYS, B, true, false, LIGHT> : (const void*)k_search<HASHED_KEYS, B, false, true, LIGHT>;
    MK_FN(256) MK_FN(512)
#undef MK_FN
    return nullptr;
}

static cudaError_t prepare(const void* f, size_t dyn) {
    return cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)dyn);
}

cudaError_t search_kernel(bool incr, uint32_t kpt, uint32_t block, bool light, uint32_t dfa_smem, uint32_t table_smem,
                          const void** func, size_t* dyn) {
    const uint32_t tsm = incr ? 0 : table_smem;
    const void* f = tsm ? stab_kernel_of(kpt, block)
                    : light ? kernel_of<true>(incr, block)
                            : kernel_of<false>(incr, block);
    // a comb table takes the shared memory of DFA tables
    if (!f || dfa_smem > DFA_SMEM_MAX || (tsm && dfa_smem)) return cudaErrorInvalidValue;
    *func = f;
    *dyn = dyn_bytes(incr, block, tsm) + dfa_smem;
    return prepare(f, *dyn);
}

cudaError_t launch_search(const KeyLaunch& L, uint32_t kpt, uint32_t block, uint32_t grid, cudaStream_t st) {
    const bool incr = L.seed_src == SEED_INCREMENTAL;
    if (incr && !L.incr) return cudaErrorInvalidValue;
    const void* f = nullptr;
    size_t dyn = 0;
    cudaError_t e = search_kernel(incr, kpt, block, L.light, L.dfa_smem, L.table_smem, &f, &dyn);
    if (e != cudaSuccess) return e;
    void* args[] = {const_cast<KeyLaunch*>(&L)};
    return cudaLaunchKernel(f, dim3(grid), dim3(block), args, dyn, st);
}

cudaError_t search_occupancy(uint32_t kpt, uint32_t block, uint32_t table_smem, int* blocks_per_sm) {
    const void* f = nullptr;
    size_t dyn = 0;
    cudaError_t e = search_kernel(false, kpt, block, false, 0, table_smem, &f, &dyn);
    if (e != cudaSuccess) return e;
    return cudaOccupancyMaxActiveBlocksPerMultiprocessor(blocks_per_sm, f, (int)block, dyn);
}

cudaError_t search_dfa_room(bool incr, uint32_t block, uint32_t ctas, uint32_t* room) {
    const void* f = nullptr;
    size_t dyn = 0;
    *room = 0;
    cudaError_t e = search_kernel(incr, 0, block, false, 0, 0, &f, &dyn);
    cudaFuncAttributes fa{};
    if (e == cudaSuccess) e = cudaFuncGetAttributes(&fa, f);
    int device = 0, sm = 0, reserved = 0, cta_max = 0;
    if (e == cudaSuccess) e = cudaGetDevice(&device);
    if (e == cudaSuccess) e = cudaDeviceGetAttribute(&sm, cudaDevAttrMaxSharedMemoryPerMultiprocessor, device);
    if (e == cudaSuccess) e = cudaDeviceGetAttribute(&reserved, cudaDevAttrReservedSharedMemoryPerBlock, device);
    if (e == cudaSuccess) e = cudaDeviceGetAttribute(&cta_max, cudaDevAttrMaxSharedMemoryPerBlockOptin, device);
    if (e != cudaSuccess) return e;
    // a CTA's share in whole kilobytes, a multiple of the granularity shared memory is given out in
    const size_t share = std::min((size_t)cta_max, ((size_t)sm / ctas - reserved) & ~(size_t)1023);
    const size_t used = fa.sharedSizeBytes + dyn;
    if (share > used) *room = std::min(DFA_SMEM_MAX, (uint32_t)(share - used) & ~15u);
    return cudaSuccess;
}

// Keys per thread of a derive: the fewest that let one wave (512 threads per SM) hold them all, at
// most DERIVE_MAX_KEYS.  On B200 a call of 257 keys takes 72 us (61 us in the kernel) where 16 keys
// behind each other in a thread took 1286; 4099 keys 100 us against 726 at 8; 2^20 keys are 1.4 ms in
// the kernel, at 16 keys per thread.
cudaError_t launch_derive(const KeyLaunch& L, uint32_t sms, uint32_t keys, cudaStream_t st) {
    const bool incr = L.seed_src == SEED_INCREMENTAL;
    if (incr && !L.incr) return cudaErrorInvalidValue;
    uint32_t k = keys ? keys : 1;
    while (!keys && k < DERIVE_MAX_KEYS && (L.count + k - 1) / k > (uint64_t)sms * 512) k *= 2;
    const void* f = nullptr;
#define MK_FN(K) \
    if (k == K) f = incr ? (const void*)k_derive<K, true> : (const void*)k_derive<K, false>;
    MK_FN(1) MK_FN(2) MK_FN(4) MK_FN(8) MK_FN(16)
#undef MK_FN
    if (!f) return cudaErrorInvalidValue;
    const size_t dyn = incr ? 0 : DERIVE_BLOCK * sizeof(EntrySlot);
    cudaError_t e = prepare(f, dyn);
    if (e != cudaSuccess) return e;
    const uint64_t threads = (L.count + k - 1) / k;
    void* args[] = {const_cast<KeyLaunch*>(&L)};
    return cudaLaunchKernel(f, dim3((uint32_t)((threads + DERIVE_BLOCK - 1) / DERIVE_BLOCK)), dim3(DERIVE_BLOCK), args,
                            dyn, st);
}

__global__ void k_set_grams(uint32_t* bitmap, const uint32_t* grams, uint32_t n) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) atomicOr(bitmap + (grams[i] >> 5), 1u << (grams[i] & 31u));
}

cudaError_t launch_set_grams(uint32_t* bitmap, const uint32_t* grams, uint32_t n, cudaStream_t st) {
    const cudaError_t e = cudaMemsetAsync(bitmap, 0, GRAM4_WORDS * sizeof(uint32_t), st);
    if (e != cudaSuccess) return e;
    k_set_grams<<<(n + 255) / 256, 256, 0, st>>>(bitmap, grams, n);
    return cudaGetLastError();
}

cudaError_t launch_build_table(uint4* table, const CombGeom& g, const uint32_t* points, uint64_t first,
                               uint64_t count, cudaStream_t st) {
    uint32_t blocks = (uint32_t)((count + 255) / 256);
    k_build_table<<<blocks, 256, 0, st>>>(table, g, points, first, count);
    return cudaGetLastError();
}

}  // namespace mkb

namespace mkb {

// Peak of independent 32-bit multiply-adds: 8 chains per thread, no memory traffic.
__global__ void __launch_bounds__(256) k_mad_lo_peak(uint32_t iters, uint32_t x, uint32_t y, uint32_t* out) {
    uint32_t a[8];
#pragma unroll
    for (int i = 0; i < 8; i++) a[i] = threadIdx.x + i;
    for (uint32_t it = 0; it < iters; it++) {
#pragma unroll
        for (int i = 0; i < 8; i++) asm volatile("mad.lo.u32 %0, %0, %1, %2;" : "+r"(a[i]) : "r"(x), "r"(y));
    }
    uint32_t s = 0;
#pragma unroll
    for (int i = 0; i < 8; i++) s ^= a[i];
    out[(uint64_t)blockIdx.x * blockDim.x + threadIdx.x] = s;
}

// Peak of the field multiply's own instruction shape: four products a·b_i accumulated on four
// aligned pairs as one mad.lo.cc/madc.hi.cc chain (rows of even/odd accumulators, fe32.cuh), on
// four independent accumulators per thread.  The multiplier a is the accumulator's top word plus
// the iteration, so no product can be hoisted out of the loop.
__global__ void __launch_bounds__(256) k_mad_chain_peak(uint32_t iters, uint32_t seed, uint32_t* out) {
    uint32_t acc[4][9], b[4];
#pragma unroll
    for (int i = 0; i < 4; i++) b[i] = seed * (2 * i + 1) + threadIdx.x;
#pragma unroll
    for (int q = 0; q < 4; q++)
#pragma unroll
        for (int i = 0; i < 9; i++) acc[q][i] = threadIdx.x ^ (q * 9 + i);
    for (uint32_t it = 0; it < iters; it++) {
#pragma unroll
        for (int r = 0; r < 2; r++)
#pragma unroll
            for (int q = 0; q < 4; q++) {
                uint32_t* t = acc[q];
                const uint32_t a = t[8] + it;
                asm volatile(
                    "mad.lo.cc.u32 %0, %9, %10, %0;\n\t"
                    "madc.hi.cc.u32 %1, %9, %10, %1;\n\t"
                    "madc.lo.cc.u32 %2, %9, %11, %2;\n\t"
                    "madc.hi.cc.u32 %3, %9, %11, %3;\n\t"
                    "madc.lo.cc.u32 %4, %9, %12, %4;\n\t"
                    "madc.hi.cc.u32 %5, %9, %12, %5;\n\t"
                    "madc.lo.cc.u32 %6, %9, %13, %6;\n\t"
                    "madc.hi.cc.u32 %7, %9, %13, %7;\n\t"
                    "addc.u32 %8, %8, 0;\n\t"
                    : "+r"(t[0]), "+r"(t[1]), "+r"(t[2]), "+r"(t[3]), "+r"(t[4]), "+r"(t[5]), "+r"(t[6]), "+r"(t[7]),
                      "+r"(t[8])
                    : "r"(a), "r"(b[0]), "r"(b[1]), "r"(b[2]), "r"(b[3]));
            }
    }
    uint32_t s = 0;
#pragma unroll
    for (int q = 0; q < 4; q++)
#pragma unroll
        for (int i = 0; i < 9; i++) s ^= acc[q][i];
    out[(uint64_t)blockIdx.x * blockDim.x + threadIdx.x] = s;
}

// The pieces of the field multiply's instruction mix, each on 8 chains per thread (so latency
// is hidden at full occupancy and the rate is what the pipe issues).  Every product has an
// operand that changes every iteration and differs between the chains, so no product can be
// hoisted out of the loop or shared between chains:
//   KIND 0  mad.hi.u32            the high half of a 32x32 product (independent chains)
//   KIND 1  mad.wide.u32          the full 64-bit product into a 64-bit sum (independent chains)
//   KIND 2  madc.lo.cc.u32 rows   8 low halves a_i·b linked through the carry flag
//   KIND 3  madc.hi.cc.u32 rows   8 high halves a_i·b linked through the carry flag
template <int KIND>
__global__ void __launch_bounds__(256) k_imad_rate(uint32_t iters, uint32_t x, uint32_t y, uint32_t* out) {
    uint32_t a[8], t[8];
    uint64_t w[8];
#pragma unroll
    for (int i = 0; i < 8; i++) {
        a[i] = (threadIdx.x * 8 + i) * 0x9e3779b9u + x;
        t[i] = threadIdx.x ^ (i * 0x01010101u);
        w[i] = (uint64_t)a[i] << 20;
    }
    for (uint32_t it = 0; it < iters; it++) {
        if (KIND == 0) {
#pragma unroll
            for (int i = 0; i < 8; i++) asm volatile("mad.hi.u32 %0, %0, %1, %2;" : "+r"(t[i]) : "r"(a[i]), "r"(y));
        } else if (KIND == 1) {
#pragma unroll
            for (int i = 0; i < 8; i++)  // the multiplier is the sum's own low word
                asm volatile("{\n\t.reg .u32 m;\n\tcvt.u32.u64 m, %0;\n\tmad.wide.u32 %0, m, %1, %0;\n\t}"
                             : "+l"(w[i]) : "r"(a[i]));
        } else {
            const uint32_t b = t[7] + it;
            if (KIND == 2)
                asm volatile(
                    "mad.lo.cc.u32 %0, %8, %16, %0;\n\t"
                    "madc.lo.cc.u32 %1, %9, %16, %1;\n\t"
                    "madc.lo.cc.u32 %2, %10, %16, %2;\n\t"
                    "madc.lo.cc.u32 %3, %11, %16, %3;\n\t"
                    "madc.lo.cc.u32 %4, %12, %16, %4;\n\t"
                    "madc.lo.cc.u32 %5, %13, %16, %5;\n\t"
                    "madc.lo.cc.u32 %6, %14, %16, %6;\n\t"
                    "madc.lo.u32 %7, %15, %16, %7;\n\t"
                    : "+r"(t[0]), "+r"(t[1]), "+r"(t[2]), "+r"(t[3]), "+r"(t[4]), "+r"(t[5]), "+r"(t[6]), "+r"(t[7])
                    : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(a[4]), "r"(a[5]), "r"(a[6]), "r"(a[7]), "r"(b));
            else
                asm volatile(
                    "mad.hi.cc.u32 %0, %8, %16, %0;\n\t"
                    "madc.hi.cc.u32 %1, %9, %16, %1;\n\t"
                    "madc.hi.cc.u32 %2, %10, %16, %2;\n\t"
                    "madc.hi.cc.u32 %3, %11, %16, %3;\n\t"
                    "madc.hi.cc.u32 %4, %12, %16, %4;\n\t"
                    "madc.hi.cc.u32 %5, %13, %16, %5;\n\t"
                    "madc.hi.cc.u32 %6, %14, %16, %6;\n\t"
                    "madc.hi.u32 %7, %15, %16, %7;\n\t"
                    : "+r"(t[0]), "+r"(t[1]), "+r"(t[2]), "+r"(t[3]), "+r"(t[4]), "+r"(t[5]), "+r"(t[6]), "+r"(t[7])
                    : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(a[4]), "r"(a[5]), "r"(a[6]), "r"(a[7]), "r"(b));
        }
    }
    uint32_t s = 0;
#pragma unroll
    for (int i = 0; i < 8; i++) s ^= t[i] ^ (uint32_t)w[i] ^ (uint32_t)(w[i] >> 32);
    out[(uint64_t)blockIdx.x * blockDim.x + threadIdx.x] = s;
}

// Rates of the four pieces (multiply-adds per second, best of three runs of 10-30 ms each).
cudaError_t measure_imad_rates(int sms, cudaStream_t st, double rates[4]) {
    const uint32_t blocks = (uint32_t)sms * 8, threads = 256, iters = 1u << 16;
    uint32_t* out = nullptr;
    cudaError_t e = cudaMalloc(&out, sizeof(uint32_t) * blocks * threads);
    if (e != cudaSuccess) return e;
    cudaEvent_t e0, e1;
    cudaEventCreate(&e0);
    cudaEventCreate(&e1);
    auto launch = [&](int kind, uint32_t it, uint32_t x) {
        if (kind == 0) k_imad_rate<0><<<blocks, threads, 0, st>>>(it, x, 0x9876u, out);
        else if (kind == 1) k_imad_rate<1><<<blocks, threads, 0, st>>>(it, x, 0x9876u, out);
        else if (kind == 2) k_imad_rate<2><<<blocks, threads, 0, st>>>(it, x, 0x9876u, out);
        else k_imad_rate<3><<<blocks, threads, 0, st>>>(it, x, 0x9876u, out);
    };
    for (int k = 0; k < 4; k++) {
        rates[k] = 0;
        launch(k, iters / 16, 0x1234u);
    }
    for (int rep = 0; rep < 12 && e == cudaSuccess; rep++) {
        const int k = rep % 4;
        cudaEventRecord(e0, st);
        launch(k, iters, 0x1234u + rep);
        cudaEventRecord(e1, st);
        e = cudaEventSynchronize(e1);
        if (e == cudaSuccess) e = cudaGetLastError();
        float ms = 0;
        if (e == cudaSuccess) cudaEventElapsedTime(&ms, e0, e1);
        const double mads = (double)blocks * threads * iters * 8;
        if (ms > 0 && mads / (ms * 1e-3) > rates[k]) rates[k] = mads / (ms * 1e-3);
    }
    cudaEventDestroy(e0);
    cudaEventDestroy(e1);
    cudaFree(out);
    return e;
}

// Best of three timed runs (after a short warm-up) of both microbenchmarks, each about
// 10-30 ms at full occupancy: multiply-adds per second.
cudaError_t measure_mad_peaks(int sms, cudaStream_t st, double* chain_per_s, double* lo_per_s) {
    const uint32_t blocks = (uint32_t)sms * 8, threads = 256;
    uint32_t* out = nullptr;
    cudaError_t e = cudaMalloc(&out, sizeof(uint32_t) * blocks * threads);
    if (e != cudaSuccess) return e;
    cudaEvent_t e0, e1;
    cudaEventCreate(&e0);
    cudaEventCreate(&e1);
    double best_chain = 0, best_lo = 0;
    const uint32_t lo_iters = 1u << 17, chain_iters = 1u << 14;
    k_mad_lo_peak<<<blocks, threads, 0, st>>>(lo_iters / 16, 0x12345u, 0x9876u, out);
    k_mad_chain_peak<<<blocks, threads, 0, st>>>(chain_iters / 16, 0x2468u, out);
    for (int rep = 0; rep < 6 && e == cudaSuccess; rep++) {
        const bool chain = rep & 1;
        cudaEventRecord(e0, st);
        if (chain) k_mad_chain_peak<<<blocks, threads, 0, st>>>(chain_iters, 0x2468u + rep, out);
        else k_mad_lo_peak<<<blocks, threads, 0, st>>>(lo_iters, 0x12345u + rep, 0x9876u, out);
        cudaEventRecord(e1, st);
        e = cudaEventSynchronize(e1);
        if (e == cudaSuccess) e = cudaGetLastError();
        float ms = 0;
        if (e == cudaSuccess) cudaEventElapsedTime(&ms, e0, e1);
        if (ms <= 0) continue;
        const double mads = (double)blocks * threads * (chain ? (double)chain_iters * 4 * 16 : (double)lo_iters * 8);
        double& best = chain ? best_chain : best_lo;
        if (mads / (ms * 1e-3) > best) best = mads / (ms * 1e-3);
    }
    cudaEventDestroy(e0);
    cudaEventDestroy(e1);
    cudaFree(out);
    *chain_per_s = best_chain;
    *lo_per_s = best_lo;
    return e;
}

}  // namespace mkb

#include "fe26.cuh"
#include "fe51.cuh"

namespace mkb {

// Field-multiplication rate of three limb radices: four independent chains a <- a·b per
// thread, no memory traffic.  Radix 2^32 is the search kernel's field (fe32.cuh); radix
// 2^25.5 (fe26.cuh, ten limbs, 100 mad.wide products) and radix 2^51 in FP64 registers
// (fe51.cuh, five limbs, products split by fused multiply-adds) are the alternatives the
// search is not built for.  Radices 32 and 51 start from the same words and write the XOR
// of their chains' canonical words, so their outputs must agree.  RADIX 33 is radix 2^32 with
// the Karatsuba multiply (fe_mul_karatsuba), which must agree with the schoolbook form too.
template <int RADIX>
__global__ void __launch_bounds__(256) k_fe_mul_rate(uint32_t iters, uint32_t seed, uint32_t* out) {
    uint32_t sum = 0;
    uint32_t wb[8], wa[4][8];
#pragma unroll
    for (int i = 0; i < 8; i++) wb[i] = seed * (i + 3) + threadIdx.x;
#pragma unroll
    for (int q = 0; q < 4; q++)
#pragma unroll
        for (int i = 0; i < 8; i++) wa[q][i] = threadIdx.x * 7 + q * 8 + i;
    if (RADIX == 32 || RADIX == 33) {
        mk32::fe a[4], b = mk32::fe_from_words(wb);
#pragma unroll
        for (int q = 0; q < 4; q++) a[q] = mk32::fe_from_words(wa[q]);
        for (uint32_t it = 0; it < iters; it++)
#pragma unroll
            for (int q = 0; q < 4; q++) a[q] = RADIX == 33 ? mk32::fe_mul_karatsuba(a[q], b) : mk32::fe_mul(a[q], b);
#pragma unroll
        for (int q = 0; q < 4; q++) {
            uint32_t w[8];
            mk32::fe_to_words(a[q], w);
#pragma unroll
            for (int i = 0; i < 8; i++) sum ^= w[i];
        }
    } else if (RADIX == 51) {
        mk51::fe a[4], b = mk51::fe_from_words(wb);
#pragma unroll
        for (int q = 0; q < 4; q++) a[q] = mk51::fe_from_words(wa[q]);
        for (uint32_t it = 0; it < iters; it++)
#pragma unroll
            for (int q = 0; q < 4; q++) a[q] = mk51::fe_mul(a[q], b);
#pragma unroll
        for (int q = 0; q < 4; q++) {
            uint32_t w[8];
            mk51::fe_to_words(a[q], w);
#pragma unroll
            for (int i = 0; i < 8; i++) sum ^= w[i];
        }
    } else {
        mk::fe a[4], b;
#pragma unroll
        for (int i = 0; i < 10; i++) b.v[i] = (seed * (i + 3) + threadIdx.x) & 0x1ffffffu;
#pragma unroll
        for (int q = 0; q < 4; q++)
#pragma unroll
            for (int i = 0; i < 10; i++) a[q].v[i] = (threadIdx.x * 7 + q * 10 + i) & 0x1ffffffu;
        for (uint32_t it = 0; it < iters; it++)
#pragma unroll
            for (int q = 0; q < 4; q++) a[q] = mk::fe_mul(a[q], b);
#pragma unroll
        for (int q = 0; q < 4; q++)
#pragma unroll
            for (int i = 0; i < 10; i++) sum ^= a[q].v[i];
    }
    out[(uint64_t)blockIdx.x * blockDim.x + threadIdx.x] = sum;
}

cudaError_t measure_field_mul_rates(int sms, cudaStream_t st, double* radix32_per_s, double* radix26_per_s,
                                    double* radix51_per_s, bool* radix51_exact) {
    const uint32_t blocks = (uint32_t)sms * 8, threads = 256, iters = 1u << 11;
    const size_t n = (size_t)blocks * threads;
    uint32_t* out = nullptr;
    cudaError_t e = cudaMalloc(&out, sizeof(uint32_t) * n * 2);
    if (e != cudaSuccess) return e;
    cudaEvent_t e0, e1;
    cudaEventCreate(&e0);
    cudaEventCreate(&e1);
    double best[3] = {0, 0, 0};
    auto launch = [&](int r, uint32_t it, uint32_t seed, uint32_t* o) {
        if (r == 0) k_fe_mul_rate<32><<<blocks, threads, 0, st>>>(it, seed, o);
        else if (r == 1) k_fe_mul_rate<26><<<blocks, threads, 0, st>>>(it, seed, o);
        else k_fe_mul_rate<51><<<blocks, threads, 0, st>>>(it, seed, o);
    };
    for (int r = 0; r < 3; r++) launch(r, iters / 16, 5u, out);
    for (int rep = 0; rep < 9 && e == cudaSuccess; rep++) {
        const int r = rep % 3;
        cudaEventRecord(e0, st);
        launch(r, iters, 9u + rep, out);
        cudaEventRecord(e1, st);
        e = cudaEventSynchronize(e1);
        if (e == cudaSuccess) e = cudaGetLastError();
        float ms = 0;
        if (e == cudaSuccess) cudaEventElapsedTime(&ms, e0, e1);
        const double muls = (double)n * iters * 4;
        if (ms > 0 && muls / (ms * 1e-3) > best[r]) best[r] = muls / (ms * 1e-3);
    }
    // exactness of radix 2^51: the same chains in radix 2^32 end in the same words
    bool same = false;
    if (e == cudaSuccess) {
        launch(0, 97, 3u, out);
        launch(2, 97, 3u, out + n);
        e = cudaStreamSynchronize(st);
        if (e == cudaSuccess) e = cudaGetLastError();
    }
    if (e == cudaSuccess) {
        std::vector<uint32_t> h(n * 2);
        e = cudaMemcpy(h.data(), out, sizeof(uint32_t) * n * 2, cudaMemcpyDeviceToHost);
        same = e == cudaSuccess && std::equal(h.begin(), h.begin() + n, h.begin() + n);
    }
    cudaEventDestroy(e0);
    cudaEventDestroy(e1);
    cudaFree(out);
    *radix32_per_s = best[0];
    *radix26_per_s = best[1];
    *radix51_per_s = best[2];
    *radix51_exact = same;
    return e;
}

// Products of operand pairs in both radix-2^32 forms: the words (below 2^256, not reduced
// to canonical) of a[i]·b[i] mod p, schoolbook into out_s and Karatsuba into out_k.
__global__ void k_fe_mul_pairs(const uint32_t* a, const uint32_t* b, uint32_t n, uint32_t* out_s, uint32_t* out_k) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const mk32::fe x = mk32::fe_from_words(a + (size_t)i * 8), y = mk32::fe_from_words(b + (size_t)i * 8);
    const mk32::fe s = mk32::fe_mul_schoolbook(x, y), k = mk32::fe_mul_karatsuba(x, y);
#pragma unroll
    for (int w = 0; w < 8; w++) {
        out_s[(size_t)i * 8 + w] = s.v[w];
        out_k[(size_t)i * 8 + w] = k.v[w];
    }
}

cudaError_t field_mul_pairs(const uint32_t* a, const uint32_t* b, uint32_t n, uint32_t* out_s, uint32_t* out_k,
                            cudaStream_t st) {
    const size_t bytes = (size_t)n * 32;
    uint32_t* d = nullptr;
    cudaError_t e = cudaMalloc(&d, bytes * 4);
    if (e != cudaSuccess) return e;
    e = cudaMemcpyAsync(d, a, bytes, cudaMemcpyHostToDevice, st);
    if (e == cudaSuccess) e = cudaMemcpyAsync(d + (size_t)n * 8, b, bytes, cudaMemcpyHostToDevice, st);
    if (e == cudaSuccess) {
        k_fe_mul_pairs<<<(n + 255) / 256, 256, 0, st>>>(d, d + (size_t)n * 8, n, d + (size_t)n * 16,
                                                        d + (size_t)n * 24);
        e = cudaGetLastError();
    }
    if (e == cudaSuccess) e = cudaMemcpyAsync(out_s, d + (size_t)n * 16, bytes, cudaMemcpyDeviceToHost, st);
    if (e == cudaSuccess) e = cudaMemcpyAsync(out_k, d + (size_t)n * 24, bytes, cudaMemcpyDeviceToHost, st);
    if (e == cudaSuccess) e = cudaStreamSynchronize(st);
    const cudaError_t ef = cudaFree(d);
    return e != cudaSuccess ? e : ef;
}

// Rates of the two radix-2^32 multiplication forms (schoolbook and Karatsuba), measured like
// measure_field_mul_rates, and whether their chains end in the same words.
cudaError_t measure_field_mul_forms(int sms, cudaStream_t st, double* schoolbook_per_s, double* karatsuba_per_s,
                                    bool* same_words) {
    const uint32_t blocks = (uint32_t)sms * 8, threads = 256, iters = 1u << 11;
    const size_t n = (size_t)blocks * threads;
    uint32_t* out = nullptr;
    cudaError_t e = cudaMalloc(&out, sizeof(uint32_t) * n * 2);
    if (e != cudaSuccess) return e;
    cudaEvent_t e0, e1;
    cudaEventCreate(&e0);
    cudaEventCreate(&e1);
    double best[2] = {0, 0};
    auto launch = [&](int k, uint32_t it, uint32_t seed, uint32_t* o) {
        if (k == 0) k_fe_mul_rate<32><<<blocks, threads, 0, st>>>(it, seed, o);
        else k_fe_mul_rate<33><<<blocks, threads, 0, st>>>(it, seed, o);
    };
    for (int k = 0; k < 2; k++) launch(k, iters / 16, 5u, out);
    for (int rep = 0; rep < 8 && e == cudaSuccess; rep++) {
        const int k = rep & 1;
        cudaEventRecord(e0, st);
        launch(k, iters, 9u + rep, out);
        cudaEventRecord(e1, st);
        e = cudaEventSynchronize(e1);
        if (e == cudaSuccess) e = cudaGetLastError();
        float ms = 0;
        if (e == cudaSuccess) cudaEventElapsedTime(&ms, e0, e1);
        const double muls = (double)n * iters * 4;
        if (ms > 0 && muls / (ms * 1e-3) > best[k]) best[k] = muls / (ms * 1e-3);
    }
    bool same = false;
    if (e == cudaSuccess) {
        launch(0, 97, 3u, out);
        launch(1, 97, 3u, out + n);
        e = cudaStreamSynchronize(st);
        if (e == cudaSuccess) e = cudaGetLastError();
    }
    if (e == cudaSuccess) {
        std::vector<uint32_t> h(n * 2);
        e = cudaMemcpy(h.data(), out, sizeof(uint32_t) * n * 2, cudaMemcpyDeviceToHost);
        same = e == cudaSuccess && std::equal(h.begin(), h.begin() + n, h.begin() + n);
    }
    cudaEventDestroy(e0);
    cudaEventDestroy(e1);
    cudaFree(out);
    *schoolbook_per_s = best[0];
    *karatsuba_per_s = best[1];
    *same_words = same;
    return e;
}

}  // namespace mkb

// ---------------------------------------------------------------------------
// Derive without allocation: fixed device staging for mk_derive_noalloc
// ---------------------------------------------------------------------------

namespace mkb {

// Device-side staging of the public keys written by mk_derive_noalloc: 65536 keys of 32
// bytes (2 MiB).  It is a file-scope device array, so every GPU that loads this library
// holds it until the process exits, and no call has to allocate device memory for it.
static __device__ __align__(256) uint8_t g_noalloc_pubkeys[NOALLOC_MAX_KEYS * 32];

// Device address of g_noalloc_pubkeys on the current device.  The name of the array in host
// code is only a host-side stand-in; its address on the device comes from
// cudaGetSymbolAddress, which the context looks up once when it is created (with its device
// current) and keeps, so it lives and dies with the context's other device memory.
cudaError_t noalloc_staging(uint8_t** ptr) {
    void* p = nullptr;
    cudaError_t e = cudaGetSymbolAddress(&p, g_noalloc_pubkeys);
    if (e != cudaSuccess) return e;
    *ptr = static_cast<uint8_t*>(p);
    return cudaSuccess;
}

}  // namespace mkb
