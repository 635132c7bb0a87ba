// permute: the lookup-argument permutation of a prover's lookup (reference poly.h:28,
// permute.cuh:74-222; the expected output is restated in core/tests/poly.rs:569-700).
//
// Over the first `usable` rows: res_input = the input values sorted ascending by canonical value;
// res_table holds, at the first row of every run of equal values in res_input, that value
// (one occurrence taken from the table), and at every other row the table values left over,
// ascending, in row order.  Every input value must occur in the table (as the reference
// requires).  Outputs are Montgomery form.
//
// One cooperative launch does all of it: canonical keys (32 bytes); a sort of the input and of the
// table side by side (half of the CTAs each); the run starts of the sorted input, each of which
// marks the table entry it takes (binary search); two counts-and-offsets scans (run starts, free
// table entries); and the outputs.  Its steps are separated by grid barriers, where launches of
// their own (about 90 with library radix sorts) cost 0.42 ms at 4090 rows in a graph, 0.58 outside one.
//
// The sort is a least-significant-digit radix sort of (word, row) pairs, 8 bits a pass.  Which word: bit
// 253, called the sign, and the 31 bits (23 up to SHORT_WORD rows) below the highest bit in which any
// two keys, those with the sign first XORed with r, differ.  For random field elements these leave a
// handful of ties; for range tables they hold the whole value, also of negative values, which
// are r - v and have r's high words.  Ties between different keys are put right afterwards: a run of
// equal words of at most TIE_RUN rows by insertion on the full keys.  Where a longer run mixes keys (a
// few dozen small values among random ones), the runs are numbered and the rows sorted again by the
// 32 bits below the highest bit in which keys of a long run differ, then by run number, each only over
// the digits that vary.  All words are sorted by, least significant first, where they have few varying
// digits (FEW_DIGITS) or long runs are left after two such rounds.
// 2^20 rows of random elements take 0.48 ms, a range table of either sign 0.45 (1.14 where all words had
// to settle it, 0.92 with library sorts), 2^19 or 100 small values among random ones 0.80 / 0.76 (1.51 /
// 1.55, 0.98 / 1.16).
#pragma once
#include <cooperative_groups.h>
#include <cudaTypedefs.h>

namespace zk {
namespace perm {

struct __align__(16) Key {
    u32 w[8];  // canonical value, little-endian words
};

ZK_DI u32 key_sign(const Key &k) { return k.w[7] >> 29; }
ZK_DI bool key_eq(const Key &a, const Key &b) {
    u32 d = 0;
#pragma unroll
    for (int i = 0; i < 8; i++) d |= a.w[i] ^ b.w[i];
    return d == 0;
}
ZK_DI bool key_lt(const Key &a, const Key &b) {
    if (a.w[7] != b.w[7]) return a.w[7] < b.w[7];
    u32 d[8];
    return Fr::sub_raw(d, a.w, b.w) != 0;
}

constexpr u32 CTA = 1024, WARPS = CTA / 32;
constexpr u32 TIE_RUN = 16, SHORT_WORD = 1u << 16;
// A round costs its passes and the time of three to six more for the runs; all words at once need no other.
constexpr u32 FEW_DIGITS = 12, ROUNDS = 3;
// flags, zero at the start: bits in which keys (XORed with r by sign) differ, and whether signs do;
// then per round the bits in which keys of a long run differ, by array, and whether a long run mixes keys
constexpr u32 FLAGS_ALL = 9, FLAGS_ROUND = 17, FLAGS = FLAGS_ALL + ROUNDS * FLAGS_ROUND;

struct Args {
    View in[2];  // the input and the table
    View res_input, res_table;
    u32 n;
    u32 half;  // CTAs per array
    Key *keys[2], *sorted[2];
    u32 *word[2][2], *idx[2][2];  // sort pairs, ping-pong
    u32 *hist;                    // [array][CTA][256], with more than one CTA an array
    u32 *flags;                   // FLAGS words
    u32 *first, *free_;           // run starts of the sorted input; table entries not taken
    u32 *counts;                  // [2][CTA]: run starts / free entries per CTA
    u32 *left;                    // rows of the sorted table that stay, in order
    u32 *start[2];                // of the sort: rows that begin a run (`first` and `left`, written later)
    u32 *run[2];                  // of the sort: run numbers by original row
};

// the 32 bits of k below (and with) bit hb
ZK_DI u32 key_word(const Key &k, u32 hb) {
    const u32 s = hb >= 31 ? hb - 31 : 0;
    u32 lo = 0, hi = 0;
#pragma unroll
    for (u32 i = 0; i < 8; i++) {
        lo = i == (s >> 5) ? k.w[i] : lo;
        hi = i == (s >> 5) + 1 ? k.w[i] : hi;
    }
    return __funnelshift_r(lo, hi, s & 31);
}
// the sign and the 31 bits below (and with) bit hb, of a key in memory
ZK_DI u32 sign_word(const Key &k, u32 hb, u32 sign) {
    const u32 s = hb >= 30 ? hb - 30 : 0, q = s >> 5;
    const u32 bits = __funnelshift_r(k.w[q], q < 7 ? k.w[q + 1] : 0u, s & 31);
    return (sign << 31) | (bits & 0x7fffffffu);
}

ZK_DI u32 warp_incl(u32 x, u32 lane) {
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const u32 y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= (u32)o) x += y;
    }
    return x;
}
// exclusive sum over the CTA's threads; sm: WARPS words
ZK_DI u32 cta_excl(u32 v, u32 *sm, u32 &total) {
    const u32 lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    const u32 x = warp_incl(v, lane);
    if (lane == 31) sm[wid] = x;
    __syncthreads();
    if (wid == 0) sm[lane] = warp_incl(sm[lane], lane);
    __syncthreads();
    const u32 r = (wid ? sm[wid - 1] : 0) + x - v;
    total = sm[WARPS - 1];
    __syncthreads();
    return r;
}

// fn(i) for the thread's rows whose word is that of the row before, the loads of four rows in flight
template <class F>
ZK_DI void for_ties(u32 n, u32 gt, u32 gs, const u32 *word, const F &fn) {
    for (u32 i0 = gt; i0 < n; i0 += 4 * gs) {
        u32 ties = 0;
#pragma unroll
        for (u32 u = 0; u < 4; u++) {
            const u32 i = i0 + u * gs;
            const u32 w = i < n ? word[i] : 0, v = i < n && i > 0 ? word[i - 1] : ~w;
            ties |= (w == v ? 1u : 0u) << u;
        }
        for (; ties; ties &= ties - 1) fn(i0 + (__ffs(ties) - 1) * gs);
    }
}

// One stable radix pass over bits [shift, shift + 8) of an array's pairs.  Every warp owns a
// contiguous segment; whist[warp][digit] first counts it, then holds the warp's next output
// position of each digit.
ZK_DI void radix_pass(const Args &a, u32 s, u32 cta, u32 shift, u32 from, u32 *whist, u32 *sm,
                      cooperative_groups::grid_group &grid) {
    auto barrier = [&] {
        if (a.half > 1) grid.sync();
        else __syncthreads();
    };
    const u32 tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const u32 *win = a.word[s][from], *iin = a.idx[s][from];
    u32 *wout = a.word[s][from ^ 1], *iout = a.idx[s][from ^ 1];
    const u32 seg = ((a.n + a.half * WARPS - 1) / (a.half * WARPS) + 31) & ~31u;
    const u64 b64 = (u64)(cta * WARPS + warp) * seg;
    const u32 begin = b64 < a.n ? (u32)b64 : a.n, end = a.n - begin < seg ? a.n : begin + seg;
    for (u32 i = tid; i < WARPS * 256; i += CTA) whist[i] = 0;
    __syncthreads();
    u32 *mine = whist + warp * 256;
    u32 before = 0, total = 0;
    for (u32 i = begin + lane; i < end; i += 32) atomicAdd(mine + ((win[i] >> shift) & 255u), 1u);
    __syncthreads();
    if (tid < 256) {
        u32 run = 0;
        for (u32 w = 0; w < WARPS; w++) {
            const u32 c = whist[w * 256 + tid];
            whist[w * 256 + tid] = run;
            run += c;
        }
        if (a.half > 1) a.hist[(s * a.half + cta) * 256 + tid] = run;
        total = run;
    }
    if (a.half > 1) grid.sync();
    if (a.half > 1 && tid < 256) {
        total = 0;
        const u32 *h = a.hist + s * a.half * 256 + tid;
#pragma unroll 8
        for (u32 b = 0; b < a.half; b++) {
            const u32 c = h[b * 256];
            before += b < cta ? c : 0;
            total += c;
        }
    }
    u32 all;
    const u32 base = cta_excl(tid < 256 ? total : 0, sm, all) + before;
    if (tid < 256)
        for (u32 w = 0; w < WARPS; w++) whist[w * 256 + tid] += base;
    __syncthreads();
    for (u32 i0 = begin; i0 < end; i0 += 32) {  // 32 pairs at a time, in order
        const u32 i = i0 + lane;
        const bool on = i < end;
        const u32 w = on ? win[i] : 0, x = on ? iin[i] : 0;
        const u32 d = on ? (w >> shift) & 255u : 256u;
        const u32 peers = __match_any_sync(0xffffffffu, d);
        const u32 rank = __popc(peers & ((1u << lane) - 1u));
        u32 pos = on ? mine[d] + rank : 0;
        __syncwarp();
        if (on && rank == 0) mine[d] += __popc(peers);
        __syncwarp();
        if (on) {
            wout[pos] = w;
            iout[pos] = x;
        }
    }
    barrier();
}

__global__ void __launch_bounds__(CTA, 1) permute_kernel(const Args a) {
    __shared__ u32 whist[WARPS * 256];
    __shared__ u32 sm[WARPS];
    cooperative_groups::grid_group grid = cooperative_groups::this_grid();
    const u32 tid = threadIdx.x, lane = tid & 31;
    const u32 s = blockIdx.x >= a.half ? 1 : 0, cta = blockIdx.x - s * a.half;
    const u32 n = a.n;
    const u32 gt = cta * CTA + tid, gs = a.half * CTA;  // thread and stride within the array
    // ---- keys and the bits they differ in
    {
        auto signed_word = [](const Fr &x, int w) { return x.v[w] ^ (FrParams::m(w) & (0u - (x.v[7] >> 29))); };
        Fr first = Fr::load(a.in[s].at(0)).to_number();
        const u32 sign0 = first.v[7] >> 29;
        u32 k0[8], diff[9];
#pragma unroll
        for (int w = 0; w < 8; w++) k0[w] = signed_word(first, w);
#pragma unroll
        for (int w = 0; w < 9; w++) diff[w] = 0;
        for (u32 i = gt; i < n; i += gs) {
            const Fr x = Fr::load(a.in[s].at(i)).to_number();
            Key k;
#pragma unroll
            for (int w = 0; w < 8; w++) {
                k.w[w] = x.v[w];
                diff[w] |= signed_word(x, w) ^ k0[w];
            }
            diff[8] |= (x.v[7] >> 29) ^ sign0;
            a.keys[s][i] = k;
        }
#pragma unroll
        for (int w = 0; w < 9; w++) {
            const u32 d = __reduce_or_sync(0xffffffffu, diff[w]);
            if (lane == 0 && d) atomicOr(a.flags + w, d);
        }
    }
    grid.sync();
    auto read_diff = [&](const u32 *f, Key &d) {  // returns the highest bit
        u32 hb = 0;
#pragma unroll
        for (u32 w = 0; w < 8; w++) {
            d.w[w] = __ldcg(f + w);
            if (d.w[w]) hb = 32 * w + 31 - __clz(d.w[w]);
        }
        return hb;
    };
    auto barrier = [&] {  // for what an array's own CTAs exchange
        if (a.half > 1) grid.sync();
        else __syncthreads();
    };
    u32 cur = 0;
    auto sort_digits = [&](u32 vary) {
        barrier();
        for (u32 shift = 0; shift < 32; shift += 8) {
            if (!((vary >> shift) & 255u)) continue;
            radix_pass(a, s, cta, shift, cur, whist, sm, grid);
            cur ^= 1;
        }
    };
    // ---- sort by the top word
    u32 hb;  // the highest bit of the array's current word
    {
        Key all;
        hb = read_diff(a.flags, all);
        const u32 signs = __ldcg(a.flags + 8);
        const u32 drop = n <= SHORT_WORD && hb >= 30 ? 8 : 0;  // up to 2^16 rows 24 bits leave few ties
        for (u32 i = gt; i < n; i += gs) {
            const Key &x = a.keys[s][i];
            a.word[s][0][i] = sign_word(x, hb, key_sign(x)) >> drop;
            a.idx[s][0][i] = i;
        }
        sort_digits(sign_word(all, hb, signs) >> drop);
    }
    // ---- put ties right
    Key *const k = a.sorted[s];
    for (u32 round = 0;; round++) {
        u32 *word = a.word[s][cur], *idx = a.idx[s][cur];
        for (u32 i = gt; i < n; i += gs) k[i] = a.keys[s][idx[i]];
        // rows i start free; the barriers up to the take step below order this
        if (round == 0)
            for (u32 i = blockIdx.x * CTA + tid; i < n; i += gridDim.x * CTA) a.free_[i] = 1u;
        grid.sync();
        // ties: rows the sort so far has not told apart (after the first round: of one run, with equal words)
        auto tied = [&](u32 i) {
            return i > 0 && word[i] == word[i - 1] && (round == 0 || key_word(k[i], hb) == key_word(k[i - 1], hb));
        };
        u32 *flags = a.flags + FLAGS_ALL + round * FLAGS_ROUND;
        bool mixed = false;  // one witness a thread is enough
        for_ties(n, gt, gs, word, [&](u32 i) {
            if (mixed || !tied(i) || key_eq(k[i], k[i - 1])) return;
            u32 lo = i - 1, hi = i + 1;
            while (hi - lo <= TIE_RUN && tied(lo)) lo--;
            while (hi - lo <= TIE_RUN && hi < n && tied(hi)) hi++;
            mixed = hi - lo > TIE_RUN;
        });
        if (mixed) atomicOr(flags + 16, 1u);
        grid.sync();
        const bool again = __ldcg(flags + 16) != 0;
        u32 *const start = a.start[s];
        for_ties(n, gt, gs, word, [&](u32 second) {  // the second row of a short run sorts it
            const u32 i = second - 1;
            if (!tied(second) || tied(i)) return;
            u32 end = i + 2;
            while (end < n && end - i <= TIE_RUN && tied(end)) end++;
            if (end - i > TIE_RUN) return;
            for (u32 j = i + 1; j < end; j++) {
                const Key x = k[j];
                const u32 r = idx[j];
                u32 p = j;
                for (; p > i && key_lt(x, k[p - 1]); p--) {
                    k[p] = k[p - 1];
                    idx[p] = idx[p - 1];
                }
                if (p != j) {
                    k[p] = x;
                    idx[p] = r;
                }
            }
        });
        if (again)
            for (u32 i = gt; i < n; i += gs) start[i] = tied(i) ? 0u : 1u;
        grid.sync();
        if (__builtin_expect(!again, 1)) break;
        Key all;
        read_diff(a.flags, all);
        const u32 signs = __ldcg(a.flags + 8);
        u32 digits = signs;
#pragma unroll
        for (int w = 0; w < 8; w++)
#pragma unroll
            for (int b = 0; b < 32; b += 8) digits += (all.w[w] >> b) & 255u ? 1 : 0;
        if (digits <= FEW_DIGITS || round + 1 == ROUNDS) {
            for (u32 w = 0; w < 9; w++) {  // the sign last
                u32 vary = w == 8 ? signs : 0;
#pragma unroll
                for (u32 v = 0; v < 8; v++) vary = v == w ? all.w[v] : vary;
                if (!vary) continue;
                for (u32 i = gt; i < n; i += gs) {
                    const Key &x = a.keys[s][a.idx[s][cur][i]];
                    a.word[s][cur][i] = w == 8 ? key_sign(x) : x.w[w];
                }
                sort_digits(vary);
            }
            for (u32 i = gt; i < n; i += gs) k[i] = a.keys[s][a.idx[s][cur][i]];
            grid.sync();
            break;
        }
        // number the runs; the rows of a short one, in order now, are runs of their own
        for (u32 i = gt; i < n; i += gs) {
            if (!start[i] || i + 1 >= n || start[i + 1]) continue;
            u32 end = i + 2;
            while (end < n && end - i <= TIE_RUN && !start[end]) end++;
            if (end - i > TIE_RUN) continue;
            for (u32 j = i + 1; j < end; j++) start[j] = 1u;
        }
        barrier();
        const u32 share = (n + a.half - 1) / a.half;  // rows of the array's CTAs, in order
        const u64 f64 = (u64)cta * share;
        const u32 first = f64 < n ? (u32)f64 : n, last = n - first < share ? n : first + share;
        u32 starts = 0, bits[8];
#pragma unroll
        for (int w = 0; w < 8; w++) bits[w] = 0;
        for (u32 i = first + tid; i < last; i += CTA) {
            if (start[i]) {
                starts++;
                continue;
            }
#pragma unroll
            for (int w = 0; w < 8; w++) bits[w] |= k[i].w[w] ^ k[i - 1].w[w];
        }
#pragma unroll
        for (int w = 0; w < 8; w++) {
            const u32 d = __reduce_or_sync(0xffffffffu, bits[w]);
            if (lane == 0 && d) atomicOr(flags + 8 * s + w, d);
        }
        u32 total;
        cta_excl(starts, sm, total);
        if (tid == 0) a.counts[blockIdx.x] = total;
        grid.sync();
        u32 before = 0, runs0 = 0, runs1 = 0;
        for (u32 b = tid; b < 2 * a.half; b += CTA) {
            const u32 c = __ldcg(a.counts + b);
            runs0 += b < a.half ? c : 0;
            runs1 += b < a.half ? 0 : c;
            before += b >= s * a.half && b < blockIdx.x ? c : 0;
        }
        cta_excl(before, sm, before);
        cta_excl(runs0, sm, runs0);
        cta_excl(runs1, sm, runs1);
        for (u32 i0 = first; i0 < last; i0 += CTA) {
            const u32 i = i0 + tid, f = i < last ? start[i] : 0;
            const u32 p = cta_excl(f, sm, total);
            if (i < last) a.run[s][idx[i]] = before + p + f - 1;
            before += total;
        }
        // by the next word, then by run
        Key mix;
        const u32 top0 = read_diff(flags, mix);
        u32 vary = key_word(mix, top0);
        const u32 top1 = read_diff(flags + 8, mix);
        vary |= key_word(mix, top1);
        hb = s ? top1 : top0;
        for (u32 i = gt; i < n; i += gs) word[i] = key_word(a.keys[s][idx[i]], hb);
        sort_digits(vary);
        for (u32 i = gt; i < n; i += gs) a.word[s][cur][i] = a.run[s][a.idx[s][cur][i]];
        const u32 most = max(runs0, runs1) - 1;
        sort_digits(most ? 0xffffffffu >> __clz(most) : 0u);
        if (top0 <= 31 && top1 <= 31) {  // the word held all the bits that were left: no ties
            for (u32 i = gt; i < n; i += gs) k[i] = a.keys[s][a.idx[s][cur][i]];
            grid.sync();
            break;
        }
    }
    // ---- run starts of the input take a table entry each (any of equal entries)
    const Key *A = a.sorted[0], *T = a.sorted[1];
    const u32 all_t = gridDim.x * CTA, all_i = blockIdx.x * CTA + tid;
    for (u32 i = all_i; i < n; i += all_t) {
        const Key goal = A[i];
        const bool head = i == 0 || !key_eq(goal, A[i - 1]);
        a.first[i] = head ? 1u : 0u;
        if (!head) continue;
        u32 lo = 0, hi = n;  // first entry not less than goal
        while (lo < hi) {
            const u32 mid = (lo + hi) >> 1;
            if (key_lt(T[mid], goal)) lo = mid + 1; else hi = mid;
        }
        if (lo < n && key_eq(T[lo], goal)) a.free_[lo] = 0u;  // runs have distinct values: no race
    }
    grid.sync();
    // ---- positions: every CTA owns a contiguous range of rows
    const u32 per = (n + gridDim.x - 1) / gridDim.x;
    const u64 r64 = (u64)blockIdx.x * per;
    const u32 r0 = r64 < n ? (u32)r64 : n, r1 = n - r0 < per ? n : r0 + per;
    {
        u32 f = 0, e = 0;
        for (u32 i = r0 + tid; i < r1; i += CTA) {
            f += a.first[i];
            e += a.free_[i];
        }
        u32 tf, te;
        cta_excl(f, sm, tf);
        cta_excl(e, sm, te);
        if (tid == 0) {
            a.counts[blockIdx.x] = tf;
            a.counts[gridDim.x + blockIdx.x] = te;
        }
    }
    grid.sync();
    u32 base_f = 0, base_e = 0;
    for (u32 b = tid; b < blockIdx.x; b += CTA) {
        base_f += __ldcg(a.counts + b);
        base_e += __ldcg(a.counts + gridDim.x + b);
    }
    {
        u32 t0, t1;
        cta_excl(base_f, sm, t0);
        cta_excl(base_e, sm, t1);
        base_f = t0;
        base_e = t1;
    }
    for (u32 i0 = r0; i0 < r1; i0 += CTA) {  // the rows that stay, in order
        const u32 i = i0 + tid;
        const u32 e = i < r1 ? a.free_[i] : 0;
        u32 tot;
        const u32 p = cta_excl(e, sm, tot);
        if (e) a.left[base_e + p] = i;
        base_e += tot;
    }
    grid.sync();
    for (u32 i0 = r0; i0 < r1; i0 += CTA) {
        const u32 i = i0 + tid;
        const u32 f = i < r1 ? a.first[i] : 0;
        u32 tot;
        const u32 p = base_f + cta_excl(f, sm, tot);
        base_f += tot;
        if (i >= r1) continue;
        // a repeated row i takes leftover number (rows before i that are not run starts)
        const Key ki = A[i], kt = f ? ki : T[a.left[i - p]];
        Fr x, y;
#pragma unroll
        for (int w = 0; w < 8; w++) {
            x.v[w] = ki.w[w];
            y.v[w] = kt.w[w];
        }
        x = Fr::to_mont(x);
        x.store(a.res_input.at(i));
        (f ? x : Fr::to_mont(y)).store(a.res_table.at(i));
    }
}

// CTAs per array: enough rows for each to be worth a grid barrier (one CTA an array, up to 2048
// rows, sorts with CTA barriers alone), at most one CTA an SM in all
inline u32 ctas_per_array(u64 n) {
    const u64 want = (n + 2047) / 2048, most = (u64)num_sms() / 2;
    return (u32)(want < 1 ? 1 : (want < most ? want : most));
}

// SMs that kernels on the stream can use: those of its green context (a partition of the device) or of
// its context (fewer than the device's under an execution-resource limit)
inline cudaError_t stream_sms(cudaStream_t stream, u32 *sms) {
    int dev = 0, all = 0;
    ZK_TRY(cudaGetDevice(&dev));
    ZK_TRY(cudaDeviceGetAttribute(&all, cudaDevAttrMultiProcessorCount, dev));
    *sms = (u32)all;
    static PFN_cuStreamGetCtx_v12050 get_ctx = nullptr;
    static PFN_cuCtxGetDevResource_v12040 ctx_resource = nullptr;
    static PFN_cuGreenCtxGetDevResource_v12040 green_resource = nullptr;
    static std::once_flag once;
    std::call_once(once, [] {
        auto find = [](const char *name, unsigned version) {
            void *f = nullptr;
            cudaDriverEntryPointQueryResult q;
            const cudaError_t e = cudaGetDriverEntryPointByVersion(name, &f, version, cudaEnableDefault, &q);
            return e == cudaSuccess && q == cudaDriverEntryPointSuccess ? f : nullptr;
        };
        ctx_resource = reinterpret_cast<PFN_cuCtxGetDevResource_v12040>(find("cuCtxGetDevResource", 12040));
        green_resource = reinterpret_cast<PFN_cuGreenCtxGetDevResource_v12040>(find("cuGreenCtxGetDevResource", 12040));
        if (ctx_resource && green_resource)
            get_ctx = reinterpret_cast<PFN_cuStreamGetCtx_v12050>(find("cuStreamGetCtx", 12050));
    });
    CUcontext ctx = nullptr;
    CUgreenCtx green = nullptr;
    CUdevResource r{};
    if (get_ctx && get_ctx(stream, &ctx, &green) == CUDA_SUCCESS &&
        (green ? green_resource(green, &r, CU_DEV_RESOURCE_TYPE_SM)
               : ctx_resource(ctx, &r, CU_DEV_RESOURCE_TYPE_SM)) == CUDA_SUCCESS &&
        r.sm.smCount > 0 && r.sm.smCount < *sms)
        *sms = r.sm.smCount;
    return cudaSuccess;
}

// CTAs per array of a launch: the grid barriers need all CTAs on the stream's SMs at once
inline cudaError_t launch_ctas_per_array(u64 n, cudaStream_t stream, u32 *half) {
    u32 sms = 0;
    int per_sm = 0;
    ZK_TRY(stream_sms(stream, &sms));
    ZK_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, permute_kernel, (int)CTA, 0));
    const u32 fit = sms * (u32)per_sm / 2, want = ctas_per_array(n);
    if (fit == 0) return cudaErrorCooperativeLaunchTooLarge;
    *half = want < fit ? want : fit;
    return cudaSuccess;
}

struct Layout {
    size_t keys[2], sorted[2], word[2][2], idx[2][2], run[2], hist, flags, first, free_, counts, left, total;
};

inline Layout layout(u64 n) {
    Layout l{};
    size_t off = 0;
    auto take = [&](size_t b) {
        const size_t o = off;
        off += (b + 255) & ~(size_t)255;
        return o;
    };
    for (int s = 0; s < 2; s++) {
        l.keys[s] = take(n * sizeof(Key));
        l.sorted[s] = take(n * sizeof(Key));
        for (int i = 0; i < 2; i++) {
            l.word[s][i] = take(n * 4);
            l.idx[s][i] = take(n * 4);
        }
    }
    l.first = take(n * 4);
    l.free_ = take(n * 4);
    l.left = take(n * 4);
    const u64 ctas = 2 * ctas_per_array(n);
    l.hist = ctas > 2 ? take(ctas * 256 * 4) : 0;
    l.flags = take((FLAGS + ctas * 2) * 4);
    l.counts = l.flags + FLAGS * 4;
    for (int s = 0; s < 2; s++) l.run[s] = take(n * 4);
    l.total = off;
    return l;
}

}  // namespace perm
}  // namespace zk

extern "C" cudaError_t permute(void *temp_buffer, unsigned long *buffer_size, unsigned long usable, ConstPolyPtr input,
                               ConstPolyPtr table, PolyPtr res_input, PolyPtr res_table, cudaStream_t stream) {
    using namespace zk;
    ZK_CHECK_ARG(usable < (1ull << 31));  // row numbers and offsets are 32 bits
    const perm::Layout l = perm::layout(usable);
    if (temp_buffer == nullptr) {
        ZK_CHECK_ARG(buffer_size != nullptr);
        *buffer_size = l.total;
        return cudaSuccess;
    }
    ZK_CHECK_ARG(buffer_size == nullptr || *buffer_size >= l.total);
    ZK_CHECK_ARG(input.len == table.len && usable <= input.len && res_input.len == usable && res_table.len == usable);
    if (usable == 0) return cudaSuccess;
    perm::Args a{};
    ZK_CHECK_ARG(make_view(input, &a.in[0]) && make_view(table, &a.in[1]) && make_view(res_input, &a.res_input) &&
                 make_view(res_table, &a.res_table));
    char *base = reinterpret_cast<char *>(temp_buffer);
    auto words = [&](size_t off) { return reinterpret_cast<u32 *>(base + off); };
    a.n = (u32)usable;
    ZK_TRY(perm::launch_ctas_per_array(usable, stream, &a.half));
    for (int s = 0; s < 2; s++) {
        a.keys[s] = reinterpret_cast<perm::Key *>(base + l.keys[s]);
        a.sorted[s] = reinterpret_cast<perm::Key *>(base + l.sorted[s]);
        for (int i = 0; i < 2; i++) {
            a.word[s][i] = words(l.word[s][i]);
            a.idx[s][i] = words(l.idx[s][i]);
        }
        a.run[s] = words(l.run[s]);
    }
    a.hist = words(l.hist);
    a.flags = words(l.flags);
    a.first = words(l.first);
    a.free_ = words(l.free_);
    a.counts = words(l.counts);
    a.left = words(l.left);
    a.start[0] = a.first;
    a.start[1] = a.left;
    ZK_TRY(cudaMemsetAsync(a.flags, 0, perm::FLAGS * 4, stream));
    void *args[] = {&a};
    return cudaLaunchCooperativeKernel(reinterpret_cast<const void *>(perm::permute_kernel), dim3(2 * a.half),
                                       dim3(perm::CTA), args, 0, stream);
}

extern "C" cudaError_t zkp_permute_ctas(unsigned long usable, cudaStream_t stream, unsigned int *ctas) {
    using namespace zk;
    ZK_CHECK_ARG(ctas != nullptr && usable < (1ull << 31));
    ZK_TRY(perm::launch_ctas_per_array(usable, stream, ctas));
    *ctas *= 2;
    return cudaSuccess;
}
