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
// their own (about 90 with library radix sorts) cost 0.58 ms at 4095 rows.
//
// The sort is a least-significant-digit radix sort of (word, row) pairs, 8 bits a pass.  Which word:
// the 32 bits (24 up to SHORT_WORD rows) below the highest bit in which any two keys differ.  For random field
// elements these leave a handful of ties, for small values (range tables) they hold the whole
// value.  Ties between different keys are put right afterwards: a run of equal words of at most
// TIE_RUN rows by insertion on the full keys; if a longer run mixes keys, the sort runs again
// over all eight words, least significant first (digits that no two keys differ in are skipped in
// every case).  So any values sort exactly, and the usual ones in three or four passes instead of 32.
#pragma once
#include <cooperative_groups.h>

namespace zk {
namespace perm {

struct __align__(16) Key {
    u32 w[8];  // canonical value, little-endian words
};

ZK_DI bool key_eq(const Key &a, const Key &b) {
    u32 d = 0;
#pragma unroll
    for (int i = 0; i < 8; i++) d |= a.w[i] ^ b.w[i];
    return d == 0;
}
ZK_DI bool key_lt(const Key &a, const Key &b) {
#pragma unroll
    for (int i = 7; i >= 0; i--)
        if (a.w[i] != b.w[i]) return a.w[i] < b.w[i];
    return false;
}

constexpr u32 CTA = 1024, WARPS = CTA / 32;
constexpr u32 TIE_RUN = 16, SHORT_WORD = 1u << 16;

struct Args {
    View in[2];  // the input and the table
    View res_input, res_table;
    u32 n;
    u32 half;  // CTAs per array
    Key *keys[2], *sorted[2];
    u32 *word[2][2], *idx[2][2];  // sort pairs, ping-pong
    u32 *hist;                    // [array][CTA][256], with more than one CTA an array
    u32 *diff;                    // 8 words: bits in which keys differ; word 8: mixed long run seen
    u32 *first, *free_;           // run starts of the sorted input; table entries not taken
    u32 *counts;                  // [2][CTA]: run starts / free entries per CTA
    u32 *left;                    // rows of the sorted table that stay, in order
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
    // ---- canonical keys and the bits they differ in
    {
        const Key k0 = [&] {
            const Fr x = Fr::load(a.in[s].at(0)).to_number();
            Key k;
#pragma unroll
            for (int w = 0; w < 8; w++) k.w[w] = x.v[w];
            return k;
        }();
        u32 diff[8];
#pragma unroll
        for (int w = 0; w < 8; w++) diff[w] = 0;
        for (u32 i = gt; i < n; i += gs) {
            const Fr x = Fr::load(a.in[s].at(i)).to_number();
            Key k;
#pragma unroll
            for (int w = 0; w < 8; w++) {
                k.w[w] = x.v[w];
                diff[w] |= x.v[w] ^ k0.w[w];
            }
            a.keys[s][i] = k;
        }
#pragma unroll
        for (int w = 0; w < 8; w++) {
            const u32 d = __reduce_or_sync(0xffffffffu, diff[w]);
            if (lane == 0 && d) atomicOr(a.diff + w, d);
        }
    }
    grid.sync();
    u32 diff[8], hb = 0;
#pragma unroll
    for (u32 w = 0; w < 8; w++) {
        diff[w] = __ldcg(a.diff + w);
        if (diff[w]) hb = 32 * w + 31 - __clz(diff[w]);
    }
    // ---- sort by one word, or by all of them
    const u32 drop = n <= SHORT_WORD && hb >= 31 ? 8 : 0;  // up to 2^16 rows 24 bits leave few ties
    u32 cur = 0;
    bool full = false;
    for (;;) {
        for (u32 word = 0; word < (full ? 8u : 1u); word++) {
            u32 vary = 0;
            if (full) {
#pragma unroll
                for (u32 w = 0; w < 8; w++) vary = w == word ? diff[w] : vary;
                if (!vary) continue;
                for (u32 i = gt; i < n; i += gs) {
                    const u32 r = word == 0 ? i : a.idx[s][cur][i];
                    a.idx[s][cur][i] = r;
                    a.word[s][cur][i] = a.keys[s][r].w[word];
                }
            } else {
                Key d;
#pragma unroll
                for (int w = 0; w < 8; w++) d.w[w] = diff[w];
                vary = key_word(d, hb) >> drop;
                for (u32 i = gt; i < n; i += gs) {
                    a.idx[s][cur][i] = i;
                    a.word[s][cur][i] = key_word(a.keys[s][i], hb) >> drop;
                }
            }
            if (a.half > 1) grid.sync();
            else __syncthreads();
            for (u32 shift = 0; shift < 32; shift += 8) {
                if (!((vary >> shift) & 255u)) continue;
                radix_pass(a, s, cta, shift, cur, whist, sm, grid);
                cur ^= 1;
            }
        }
        for (u32 i = gt; i < n; i += gs) a.sorted[s][i] = a.keys[s][a.idx[s][cur][i]];
        // rows i start free; the barriers up to the take step below order this
        for (u32 i = blockIdx.x * CTA + tid; i < n; i += gridDim.x * CTA) a.free_[i] = 1u;
        grid.sync();
        if (full) break;
        // rows whose key differs from the one before it under an equal word
        const u32 *word = a.word[s][cur];
        bool mixed_long = false;
        for (u32 i = gt; i < n; i += gs) {
            if (i == 0 || word[i] != word[i - 1] || key_eq(a.sorted[s][i], a.sorted[s][i - 1])) continue;
            u32 lo = i, hi = i + 1;
            while (lo > 0 && word[lo - 1] == word[i] && hi - lo <= TIE_RUN) lo--;
            while (hi < n && word[hi] == word[i] && hi - lo <= TIE_RUN) hi++;
            mixed_long = mixed_long || hi - lo > TIE_RUN;
        }
        if (mixed_long) atomicOr(a.diff + 8, 1u);
        grid.sync();
        if (!__ldcg(a.diff + 8)) {
            for (u32 i = gt; i < n; i += gs) {  // the head of a short run sorts it
                if ((i > 0 && word[i] == word[i - 1]) || i + 1 >= n || word[i + 1] != word[i]) continue;
                u32 end = i + 2;
                while (end < n && word[end] == word[i] && end - i <= TIE_RUN) end++;
                if (end - i > TIE_RUN) continue;  // a long run of one key
                Key *k = a.sorted[s];
                for (u32 j = i + 1; j < end; j++) {
                    const Key x = k[j];
                    u32 p = j;
                    for (; p > i && key_lt(x, k[p - 1]); p--) k[p] = k[p - 1];
                    if (p != j) k[p] = x;
                }
            }
            grid.sync();
            break;
        }
        full = true;
        cur = 0;
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

struct Layout {
    size_t keys[2], sorted[2], word[2][2], idx[2][2], hist, diff, first, free_, counts, left, total;
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
    l.diff = take((9 + ctas * 2) * 4);
    l.counts = l.diff + 9 * 4;
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
    a.half = perm::ctas_per_array(usable);
    for (int s = 0; s < 2; s++) {
        a.keys[s] = reinterpret_cast<perm::Key *>(base + l.keys[s]);
        a.sorted[s] = reinterpret_cast<perm::Key *>(base + l.sorted[s]);
        for (int i = 0; i < 2; i++) {
            a.word[s][i] = words(l.word[s][i]);
            a.idx[s][i] = words(l.idx[s][i]);
        }
    }
    a.hist = words(l.hist);
    a.diff = words(l.diff);
    a.first = words(l.first);
    a.free_ = words(l.free_);
    a.counts = words(l.counts);
    a.left = words(l.left);
    ZK_TRY(cudaMemsetAsync(a.diff, 0, 9 * 4, stream));
    void *args[] = {&a};
    return cudaLaunchCooperativeKernel(reinterpret_cast<const void *>(perm::permute_kernel), dim3(2 * a.half),
                                       dim3(perm::CTA), args, 0, stream);
}
