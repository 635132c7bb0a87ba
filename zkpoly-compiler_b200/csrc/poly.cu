// libpoly.so: polynomial kernels over BN254 Fr for sm_100a.
//
// Replaces the reference's poly library (core/src/poly/src/poly.h:4-28, poly_basic.cuh,
// poly_eval.cuh, batched_invert.cuh, scan_mul.cuh, kate_division.cuh) behind the same C ABI.
// Temp-buffer protocol as in the reference: a null temp buffer returns the size needed.
//
// The reference builds evaluation, inversion and scans from CUB device scans with a field
// operator.  Here each of them is at most three launches of this library's own kernels: an up
// pass (every thread folds a short contiguous chunk, the CTA's threads are joined by shuffle
// scans), one CTA over the CTA results, and a down pass that walks the chunks again from their
// carry.  Each element costs one to three Montgomery products and one or two passes over HBM.
#include <cuda_runtime.h>
#include <utility>

#include "../../include/poly.h"
#include "common.cuh"
#include "curve.cuh"

namespace zk {
namespace poly {

// Threads of the sweeps' CTAs, and the most CTA results the one-CTA step takes (TOP_C a thread).
// What bounds a sweep is the length of its chain of dependent products, about 0.45 us each (a warp
// alone on its scheduler): chunk + 8 scan steps per pass.  With 256 threads an SM (two warps a
// scheduler) the chains nearly fill the multiply pipe, so the chunk is n over that many threads,
// between 2 and MAX_C elements, and longer only where the CTA results would exceed TOP_MAX.
// Fixed chunks of 32 to 64 elements and a tree of chunks of 8 above them (up to twelve launches)
// took 153 / 95 / 76 / 65 us for inversion / product scan / division (2048) / evaluation at 4095
// elements and 236 / 153 / 153 / 93 us at 2^20; this form 59 / 32 / 26 / 23 and 139 / 77 / 80 / 45
// (2^24: 1057 / 703 / 679 / 337 us, before 1049 / 760 / 751 / 359).
constexpr u32 CTA = 256, WARPS = CTA / 32;
constexpr u32 TOP_C = 16, TOP_MAX = TOP_C * CTA, MAX_C = 32;
// Up to ONE_CTA elements one CTA does everything in one launch: its chunks are longer (8 elements at
// 2048), but a chain of some 40 products is shorter than three launches (division of 2048: 25
// against 49 us; at 4095, with chunks of 16, the inversion took 87 against 62 us).
constexpr u64 ONE_CTA = 2048;
inline u32 chunk_for(u64 n) {
    u32 c = 2;
    if (n <= ONE_CTA) {
        while (n > (u64)CTA * c) c *= 2;
        return c;
    }
    while (c < MAX_C && n > (u64)num_sms() * CTA * c) c *= 2;
    while (c < (1u << 30) && n > (u64)TOP_MAX * CTA * c) c *= 2;
    return c;
}
// elements a thread of the one-CTA step
inline u32 top_chunk(u64 m) {
    u32 c = 1;
    while (m > (u64)CTA * c) c *= 2;
    return c;
}
inline u32 log2_of(u32 c) { return 31 - __builtin_clz(c); }
// the sweeps that walk their elements twice: up to four elements are one chunk, walked by one thread
inline u32 walk_chunk_for(u64 n) { return n <= 4 ? 4 : chunk_for(n); }
// One warp where its lanes hold all the chunks (SMALL kernels).  Its scans then stop at the chunks there
// are, which for a handful of elements is most of the chain (1 / 8 elements through a whole CTA's
// steps, by one thread, and here: product scan 7.3 / 8.4, 2.3 / 8.1 and 2.1 / 4.2 us, division 13.5 / 14.6,
// 2.0 / 7.0 and 2.2 / 5.2, inversion 45 / 48, 35 / 49 and 21 / 26).
inline bool one_warp(u64 n, u32 c) { return n <= 32ull * c; }
// an empty polynomial counts as one CTA, so that no size query answers 0 (a caller's buffer of 0 bytes
// is a null pointer, which asks for the size again)
inline u64 ctas_for(u64 n, u32 c) { return n ? (n + (u64)CTA * c - 1) / ((u64)CTA * c) : 1; }

inline u32 grid_for(u64 items, u32 block, u32 per_sm = 16) {
    const u64 b = (items + block - 1) / block;
    const u64 cap = (u64)num_sms() * per_sm;
    return (u32)(b < cap ? (b == 0 ? 1 : b) : cap);
}

inline View plain_view(void *p, u64 n) {
    View v;
    v.base = reinterpret_cast<u32 *>(p);
    v.off = 0;
    v.whole = n ? n : 1;
    v.len = n;
    return v;
}

// ------------------------------------------------------------------ elementwise
enum Op : u32 { OP_ADD = 0, OP_SUB = 1, OP_MUL = 2, OP_SUBR = 3, OP_SQR = 4 };

// dst[i] = a[i] op b[i] for i < len; dst[i] = a[i] (or -a[i] for reversed subtraction) for
// len <= i < upper (poly_basic.cuh:4-65: the longer operand passes through)
__global__ void __launch_bounds__(256) binary_kernel(View dst, View a, View b, u64 len, u64 upper, u32 op) {
    const u64 stride = (u64)gridDim.x * blockDim.x;
    for (u64 i = (u64)blockIdx.x * blockDim.x + threadIdx.x; i < upper; i += stride) {
        Fr x = Fr::load(a.at(i)), r;
        if (i < len) {
            Fr y = Fr::load(b.at(i));
            switch (op) {
                case OP_ADD: r = Fr::add_c(x, y); break;
                case OP_SUB: r = Fr::sub_c(x, y); break;
                case OP_SUBR: r = Fr::sub_c(y, x); break;
                case OP_SQR: r = Fr::sqr(x).canonical(); break;
                default: r = Fr::mul(x, y).canonical(); break;
            }
        } else {
            r = op == OP_SUBR ? Fr::neg(x).canonical() : x;
        }
        r.store(dst.at(i));
    }
}

// coef = true: value at index 0, zero elsewhere (poly_set_coef); else value everywhere
__global__ void __launch_bounds__(256) fill_kernel(View dst, u64 n, u32 kind, bool coef) {
    const u64 stride = (u64)gridDim.x * blockDim.x;
    for (u64 i = (u64)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += stride) {
        Fr v = (kind == 1 && (!coef || i == 0)) ? Fr::one() : Fr::zero();
        v.store(dst.at(i));
    }
}

// one warp
__global__ void scalar_kernel(u32 *target, u64 exp, u32 kind) {
    const Fr x = Fr::load(target);
    const Fr r = kind == 0 ? inv_binary_quad<FrParams>(x) : Fr::pow_u64(x, exp).canonical();
    __syncwarp();
    if (threadIdx.x == 0) r.store(target);
}

// ------------------------------------------------------------------ CTA-wide steps
ZK_DI Fr lane_get(const Fr &x, u32 src) {
    Fr r;
#pragma unroll
    for (int w = 0; w < 8; w++) r.v[w] = __shfl_sync(0xffffffffu, x.v[w], src);
    return r;
}
ZK_DI Fr pick(bool c, const Fr &a, const Fr &b) {
    Fr r;
#pragma unroll
    for (int w = 0; w < 8; w++) r.v[w] = c ? a.v[w] : b.v[w];
    return r;
}

// lad[b] = base^(2^b) for b < count (<= 32), by warp 0: lane b squares b times
ZK_DI void power_ladder(const Fr &base, u32 count, u32 *lad) {
    if (threadIdx.x >= 32) return;
    Fr x = base;
#pragma unroll 1
    for (u32 b = 0; b + 1 < count; b++) x = pick(threadIdx.x > b, Fr::sqr(x), x);
    if (threadIdx.x < count) x.store(lad + threadIdx.x * 8);
}

// exclusive product of the threads before (e) and, with BOTH, after (f); sm: WARPS elements.  The
// two directions' products of a step are independent.
template <bool BOTH>
ZK_DI void lane_products(Fr &x, Fr &y, u32 lane, u32 width) {
#pragma unroll 1
    for (u32 d = 1; d < width; d <<= 1) {
        const Fr a = Fr::mul(x, lane_get(x, lane - d));
        if (BOTH) y = pick(lane + d < width, Fr::mul(y, lane_get(y, lane + d)), y);
        x = pick(lane >= d, a, x);
    }
}
template <bool BOTH>
ZK_DI void cta_products(const Fr &v, u32 *sm, Fr &e, Fr &f, Fr &total) {
    const u32 lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    Fr x = v, y = v;
    lane_products<BOTH>(x, y, lane, 32);
    if (lane == 31) x.store(sm + warp * 8);
    __syncthreads();
    Fr wx = lane < WARPS ? Fr::load(sm + lane * 8) : Fr::one(), wy = wx;
    lane_products<BOTH>(wx, wy, lane, WARPS);
    total = lane_get(wx, WARPS - 1);
    const Fr bx = lane_get(wx, warp - 1);
    e = pick(lane > 0, lane_get(x, lane - 1), Fr::one());
    if (warp > 0) e = Fr::mul(e, bx);
    if (BOTH) {
        const Fr by = lane_get(wy, warp + 1);
        f = pick(lane < 31, lane_get(y, lane + 1), Fr::one());
        if (warp + 1 < WARPS) f = Fr::mul(f, by);
    }
    __syncthreads();
}

// the same for a CTA of one warp whose first `chunks` lanes hold values (ones after them)
template <bool BOTH>
ZK_DI void warp_products(const Fr &v, u32 chunks, Fr &e, Fr &f, Fr &total) {
    const u32 lane = threadIdx.x & 31;
    Fr x = v, y = v;
    lane_products<BOTH>(x, y, lane, chunks);
    total = lane_get(x, chunks - 1);
    e = pick(lane > 0, lane_get(x, lane - 1), Fr::one());
    if (BOTH) f = pick(lane < 31, lane_get(y, lane + 1), Fr::one());
}

// ------------------------------------------------------------------ evaluation
// out[cta] = sum over the CTA's CTA * c coefficients a_i X^(i - first); next_base = X^(CTA c), the
// point of the next level.  A thread's chunk is a Horner chain, the chunks are joined by shuffles
// with X^c, X^2c, ... from the ladder.
__global__ void __launch_bounds__(CTA) eval_kernel(View in, u64 n, const u32 *base, u32 c, u32 logc, u32 *out,
                                                   u32 *next_base) {
    __shared__ __align__(16) u32 lad[32 * 8];
    __shared__ __align__(16) u32 sm[WARPS * 8];
    const u32 lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const Fr X = Fr::load(base);
    power_ladder(X, logc + 9, lad);
    const u64 start = ((u64)blockIdx.x * CTA + threadIdx.x) * c;
    Fr h = Fr::zero();
    if (start < n) {
        const u64 end = start + c < n ? start + c : n;
        h = Fr::load(in.at(end - 1));
#pragma unroll 4
        for (u64 i = end - 1; i-- > start;) h = Fr::add(Fr::mul(h, X), Fr::load(in.at(i)));
    }
    __syncthreads();
#pragma unroll 1
    for (u32 s = 0; s < 5; s++) h = Fr::add(Fr::mul(lane_get(h, lane + (1u << s)), Fr::load(lad + (logc + s) * 8)), h);
    if (lane == 0) h.store(sm + warp * 8);
    __syncthreads();
    if (warp) return;
    h = lane < WARPS ? Fr::load(sm + lane * 8) : Fr::zero();
#pragma unroll 1
    for (u32 s = 0; s < 3; s++)
        h = Fr::add(Fr::mul(lane_get(h, lane + (1u << s)), Fr::load(lad + (logc + 5 + s) * 8)), h);
    if (lane == 0) {
        h.canonical().store(out + (u64)blockIdx.x * 8);
        if (blockIdx.x == 0 && next_base) Fr::load(lad + (logc + 8) * 8).store(next_base);
    }
}

// ------------------------------------------------------------------ product scan
// A pass over few values a thread folds its chunk again in the down pass instead of keeping one
// value a chunk (ex null): the chunk results of short chunks would not fit the scratch the tree of
// chunks needed, and callers may hold scratch of that size.
ZK_DI Fr chunk_product(const View &in, u64 n, u64 start, u32 c) {
    if (start >= n) return Fr::one();
    const u64 end = start + c < n ? start + c : n;
    Fr acc = Fr::load(in.at(start));
#pragma unroll 4
    for (u64 i = start + 1; i < end; i++) acc = Fr::mul(acc, Fr::load(in.at(i)));
    return acc;
}
// up: ex[t] = product of the CTA's chunks before chunk t, tot[cta] = the CTA's product
__global__ void __launch_bounds__(CTA) scan_up_kernel(View in, u64 n, u32 c, u32 *ex, u32 *tot) {
    __shared__ __align__(16) u32 sm[WARPS * 8];
    const u64 t = (u64)blockIdx.x * CTA + threadIdx.x, start = t * c;
    Fr e, f, total;
    cta_products<false>(chunk_product(in, n, start, c), sm, e, f, total);
    if (ex && start < n) e.store(ex + t * 8);
    if (threadIdx.x == 0) total.store(tot + (u64)blockIdx.x * 8);
}
// exclusive product scan of at most TOP_MAX values in place (one CTA)
__global__ void __launch_bounds__(CTA) scan_top_kernel(u32 *vals, u32 m, u32 c) {
    __shared__ __align__(16) u32 sm[WARPS * 8];
    const u32 start = threadIdx.x * c, end = start + c < m ? start + c : m;
    Fr acc = Fr::one();
    for (u32 i = start; i < end; i++) acc = Fr::mul(acc, Fr::load(vals + (u64)i * 8));
    Fr e, f, total;
    cta_products<false>(acc, sm, e, f, total);
    for (u32 i = start; i < end; i++) {
        const Fr v = Fr::load(vals + (u64)i * 8);
        e.store(vals + (u64)i * 8);
        e = Fr::mul(e, v);
    }
}
// cta_ex null: a single CTA; SMALL: it is one warp
template <bool SMALL>
__global__ void __launch_bounds__(CTA) scan_down_kernel(View data, u64 n, u32 c, const u32 *ex, const u32 *cta_ex) {
    __shared__ __align__(16) u32 sm[WARPS * 8];
    const u64 t = (u64)blockIdx.x * CTA + threadIdx.x, start = t * c;
    Fr acc;
    if (ex) {
        if (start >= n) return;
        acc = Fr::load(ex + t * 8);
    } else {
        Fr f, total;
        if (!SMALL) cta_products<false>(chunk_product(data, n, start, c), sm, acc, f, total);
        else if (n <= c) acc = Fr::one();
        else warp_products<false>(chunk_product(data, n, start, c), (u32)((n + c - 1) / c), acc, f, total);
        if (start >= n) return;
    }
    if (cta_ex) acc = Fr::mul(acc, Fr::load(cta_ex + (u64)blockIdx.x * 8));
    const u64 end = start + c < n ? start + c : n;
#pragma unroll 4
    for (u64 i = start; i < end; i++) {
        u32 *p = data.at(i);
        acc = Fr::mul(acc, Fr::load(p));
        acc.canonical().store(p);
    }
}

// ------------------------------------------------------------------ batched inversion
// Montgomery's trick: up, prefix[i] = running product inside the chunk (zeros skipped) for all but
// its last element, whose place takes the product of the CTA's other chunks; tot[cta] = the CTA's
// product; one CTA inverts the product
// of all CTA products and hands every CTA its inverse; down, a chunk starts from
// inv_tot[cta] prefix[last] = (chunk product)^-1 and walks backwards.
__global__ void __launch_bounds__(CTA) inv_up_kernel(View in, u64 n, u32 c, u32 *prefix, u32 *tot) {
    __shared__ __align__(16) u32 sm[WARPS * 8];
    const u64 t = (u64)blockIdx.x * CTA + threadIdx.x, start = t * c;
    Fr acc = Fr::one();
    if (start < n) {
        const u64 end = start + c < n ? start + c : n;
#pragma unroll 4
        for (u64 i = start; i < end; i++) {
            const Fr a = Fr::load(in.at(i));
            acc = pick(a.is_zero(), acc, Fr::mul(acc, a));
            if (i + 1 < end) acc.store(prefix + i * 8);
        }
    }
    Fr e, f, total;
    cta_products<true>(acc, sm, e, f, total);
    if (start < n) Fr::mul(e, f).store(prefix + ((start + c < n ? start + c : n) - 1) * 8);
    if (threadIdx.x == 0) total.store(tot + (u64)blockIdx.x * 8);
}
// inverses of at most TOP_MAX non-zero values in place (one CTA); prefix: m elements
__global__ void __launch_bounds__(CTA) inv_top_kernel(u32 *vals, u32 m, u32 c, u32 *prefix) {
    __shared__ __align__(16) u32 sm[WARPS * 8];
    const u32 start = threadIdx.x * c, end = start + c < m ? start + c : m;
    Fr acc = Fr::one();
    for (u32 i = start; i < end; i++) {
        acc.store(prefix + (u64)i * 8);
        acc = Fr::mul(acc, Fr::load(vals + (u64)i * 8));
    }
    Fr e, f, total;
    cta_products<true>(acc, sm, e, f, total);
    if (threadIdx.x < 32) {
        const Fr inv_all = inv_binary_quad<FrParams>(total);
        if (threadIdx.x == 0) inv_all.store(sm);
    }
    __syncthreads();
    Fr inv = Fr::mul(Fr::load(sm), Fr::mul(e, f));
    for (u32 i = end; i-- > start;) {
        const Fr v = Fr::load(vals + (u64)i * 8);
        Fr::mul(inv, Fr::load(prefix + (u64)i * 8)).store(vals + (u64)i * 8);
        inv = Fr::mul(inv, v);
    }
}
// all of it for one CTA's elements (SMALL: a CTA of one warp); prefix: n elements
template <bool SMALL>
__global__ void __launch_bounds__(CTA) inv_one_kernel(View data, u32 n, u32 c, u32 *prefix) {
    __shared__ __align__(16) u32 sm[WARPS * 8];
    const u32 start = threadIdx.x * c, end = start + c < n ? start + c : n;
    Fr acc = Fr::one();
#pragma unroll 2
    for (u32 i = start; i < end; i++) {
        const Fr a = Fr::load(data.at(i));
        acc.store(prefix + (u64)i * 8);
        acc = pick(a.is_zero(), acc, Fr::mul(acc, a));
    }
    Fr e, f, total;
    const bool alone = SMALL && n <= c;  // one chunk: nothing before or after it
    if (!SMALL) cta_products<true>(acc, sm, e, f, total);
    else warp_products<true>(acc, (n + c - 1) / c, e, f, total);
    const Fr ef = alone ? Fr::one() : Fr::mul(e, f);
    if (threadIdx.x < 32) {
        const Fr inv_all = inv_binary_quad<FrParams>(total);
        if (threadIdx.x == 0) inv_all.store(sm);
    }
    __syncthreads();
    Fr inv = alone ? Fr::load(sm) : Fr::mul(Fr::load(sm), ef);
#pragma unroll 2
    for (u32 i = end; i-- > start;) {
        u32 *p = data.at(i);
        const Fr a = Fr::load(p);
        if (a.is_zero()) continue;
        const Fr r = Fr::mul(inv, Fr::load(prefix + (u64)i * 8));
        inv = Fr::mul(inv, a);
        r.canonical().store(p);
    }
}
__global__ void __launch_bounds__(CTA) inv_down_kernel(View data, u64 n, u32 c, const u32 *prefix,
                                                       const u32 *inv_tot) {
    const u64 t = (u64)blockIdx.x * CTA + threadIdx.x, start = t * c;
    if (start >= n) return;
    const u64 end = start + c < n ? start + c : n;
    Fr inv = Fr::mul(Fr::load(prefix + (end - 1) * 8), Fr::load(inv_tot + (u64)blockIdx.x * 8));
#pragma unroll 2
    for (u64 i = end; i-- > start;) {
        u32 *p = data.at(i);
        const Fr a = Fr::load(p);
        if (a.is_zero()) continue;
        const Fr before = i > start ? Fr::load(prefix + (i - 1) * 8) : Fr::one();
        const Fr r = Fr::mul(inv, before);
        inv = Fr::mul(inv, a);
        r.canonical().store(p);
    }
}

// ------------------------------------------------------------------ kate division
// q[i] = sum_{j > i} p_j b^(j-i-1), i.e. q[i] = p[i+1] + b q[i+1] with q[n-1] = 0
// (kate_division.cuh:1-85, halo2 kate_division).  A chunk's carry is q at the first index after it.
// up: the chunk-local value at the chunk's start (Horner from its top), then a suffix scan over
// the CTA with b^c, b^2c, ... gives carry[t], the carry from the CTA's own later chunks, and
// tot[cta], the value at the CTA's start; one CTA turns those into the carry into every CTA; down
// adds b^(c (chunks to the CTA's end)) times that carry and walks each chunk downwards.
// tab (written by CTA 0): b^(c j) for j < 32, then b^(32 c j) for j < WARPS, then b^(CTA c).
constexpr u32 TAB = 32 + WARPS + 1;

// lad: b^(2^k), k < logc + 9; pw[j] = b^(c j), j < 32 (warp 0)
ZK_DI void chunk_powers(const u32 *lad, u32 logc, u32 *pw) {
    if (threadIdx.x >= 32) return;
    Fr x = Fr::one();
#pragma unroll 1
    for (u32 k = 0; k < 5; k++)
        x = pick((threadIdx.x >> k) & 1, Fr::mul(x, Fr::load(lad + (logc + k) * 8)), x);
    x.store(pw + threadIdx.x * 8);
}
// carry into the thread's chunk from the CTA's later chunks, for chunk-local values v; total = the
// value at the CTA's start (in lane 0 of warp 0)
ZK_DI Fr cta_suffix(Fr v, const u32 *lad, u32 logc, const u32 *pw, u32 *sm, Fr &total) {
    const u32 lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll 1
    for (u32 s = 0; s < 5; s++) {
        const Fr x = Fr::add(Fr::mul(lane_get(v, lane + (1u << s)), Fr::load(lad + (logc + s) * 8)), v);
        v = pick(lane + (1u << s) < 32, x, v);
    }
    if (lane == 0) v.store(sm + warp * 8);
    __syncthreads();
    Fr w = lane < WARPS ? Fr::load(sm + lane * 8) : Fr::zero();
#pragma unroll 1
    for (u32 s = 0; s < 3; s++) {
        const Fr x = Fr::add(Fr::mul(lane_get(w, lane + (1u << s)), Fr::load(lad + (logc + 5 + s) * 8)), w);
        w = pick(lane + (1u << s) < WARPS, x, w);
    }
    total = w;
    const Fr next = pick(warp + 1 < WARPS, lane_get(w, warp + 1), Fr::zero());
    const Fr after = pick(lane < 31, lane_get(v, lane + 1), Fr::zero());
    return Fr::add(Fr::mul(Fr::load(pw + (31 - lane) * 8), next), after);
}

// the same for a CTA of one warp whose first `chunks` lanes hold values (zeros after them)
ZK_DI Fr warp_suffix(Fr v, const u32 *lad, u32 logc, u32 chunks) {
    const u32 lane = threadIdx.x & 31;
#pragma unroll 1
    for (u32 s = 0; (1u << s) < chunks; s++) {
        const Fr x = Fr::add(Fr::mul(lane_get(v, lane + (1u << s)), Fr::load(lad + (logc + s) * 8)), v);
        v = pick(lane + (1u << s) < 32, x, v);
    }
    return pick(lane < 31, lane_get(v, lane + 1), Fr::zero());
}

// q at `start` from the chunk's own terms p[start + 1 .. end]
ZK_DI Fr chunk_local(const View &p, u64 n, u64 start, u32 c, const Fr &B) {
    if (start >= n) return Fr::zero();
    const u64 end = start + c < n ? start + c : n;
    Fr acc = end < n ? Fr::load(p.at(end)) : Fr::zero();
#pragma unroll 4
    for (u64 j = end - 1; j > start; j--) acc = Fr::add(Fr::mul(acc, B), Fr::load(p.at(j)));
    return acc;
}
__global__ void __launch_bounds__(CTA) kate_up_kernel(View p, u64 n, const u32 *b, u32 c, u32 logc, u32 *carry,
                                                      u32 *tot, u32 *tab) {
    __shared__ __align__(16) u32 lad[32 * 8], pw[32 * 8], sm[WARPS * 8];
    const Fr B = Fr::load(b);
    power_ladder(B, logc + 9, lad);
    __syncwarp();
    chunk_powers(lad, logc, pw);
    const u64 t = (u64)blockIdx.x * CTA + threadIdx.x, start = t * c;
    const Fr acc = chunk_local(p, n, start, c, B);
    __syncthreads();
    Fr total;
    const Fr in = cta_suffix(acc, lad, logc, pw, sm, total);
    if (carry && start < n) in.store(carry + t * 8);
    if (threadIdx.x == 0) total.store(tot + (u64)blockIdx.x * 8);
    if (blockIdx.x == 0 && threadIdx.x < 32) {
        const u32 lane = threadIdx.x;
        Fr::load(pw + lane * 8).store(tab + lane * 8);
        Fr x = Fr::one();
#pragma unroll 1
        for (u32 k = 0; k < 3; k++) x = pick((lane >> k) & 1, Fr::mul(x, Fr::load(lad + (logc + 5 + k) * 8)), x);
        if (lane < WARPS) x.store(tab + (32 + lane) * 8);
        if (lane == 0) Fr::load(lad + (logc + 8) * 8).store(tab + (32 + WARPS) * 8);
    }
}
// vals[i] <- the carry into CTA i: x_i = vals[i+1] + base x_(i+1), 0 for the last (one CTA)
__global__ void __launch_bounds__(CTA) kate_top_kernel(u32 *vals, u32 m, const u32 *base, u32 c, u32 logc) {
    __shared__ __align__(16) u32 lad[32 * 8], pw[32 * 8], sm[WARPS * 8];
    const Fr B = Fr::load(base);
    power_ladder(B, logc + 9, lad);
    __syncwarp();
    chunk_powers(lad, logc, pw);
    const u32 start = threadIdx.x * c, end = start + c < m ? start + c : m;
    Fr acc = Fr::zero();
    for (u32 i = end; i-- > start;) acc = Fr::add(Fr::mul(acc, B), Fr::load(vals + (u64)i * 8));
    __syncthreads();
    Fr total;
    Fr in = cta_suffix(acc, lad, logc, pw, sm, total);
    for (u32 i = end; i-- > start;) {
        const Fr v = Fr::load(vals + (u64)i * 8);
        in.store(vals + (u64)i * 8);
        in = Fr::add(Fr::mul(in, B), v);
    }
}
// carry null: recomputed as in the up pass (see the product scan); tab null: a single CTA; SMALL: it is
// one warp
template <bool SMALL>
__global__ void __launch_bounds__(CTA) kate_down_kernel(View p, View q, u64 n, const u32 *b, u32 c, u32 logc,
                                                        const u32 *carry, const u32 *cta_in, const u32 *tab) {
    __shared__ __align__(16) u32 lad[32 * 8], pw[32 * 8], sm[WARPS * 8];
    const u64 t = (u64)blockIdx.x * CTA + threadIdx.x, start = t * c;
    const u32 lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const Fr B = Fr::load(b);
    Fr acc;
    if (carry) {
        if (start >= n) return;
        acc = Fr::load(carry + t * 8);
    } else if (SMALL) {
        acc = Fr::zero();
        if (n > c) {
            const u32 chunks = (u32)((n + c - 1) / c);
            power_ladder(B, logc + 32 - __clz(chunks - 1), lad);  // up to b^(c 2^(steps - 1))
            __syncwarp();
            acc = warp_suffix(chunk_local(p, n, start, c, B), lad, logc, chunks);
        }
        if (start >= n) return;
    } else {
        power_ladder(B, logc + 9, lad);
        __syncwarp();
        chunk_powers(lad, logc, pw);
        const Fr local = chunk_local(p, n, start, c, B);
        __syncthreads();
        Fr total;
        acc = cta_suffix(local, lad, logc, pw, sm, total);
        if (start >= n) return;
    }
    if (tab) {
        const Fr z = Fr::mul(Fr::load(cta_in + (u64)blockIdx.x * 8), Fr::load(tab + (32 + WARPS - 1 - warp) * 8));
        acc = Fr::add(Fr::mul(z, Fr::load(tab + (31 - lane) * 8)), acc);
    }
    const u64 end = start + c < n ? start + c : n;
#pragma unroll 4
    for (u64 i = end; i-- > start;) {
        const u64 j = i + 1;
        const Fr pj = j < n ? Fr::load(p.at(j)) : Fr::zero();
        acc = Fr::add(Fr::mul(acc, B), pj);
        acc.canonical().store(q.at(i));
    }
}

inline size_t al(size_t x) { return (x + 255) & ~(size_t)255; }

}  // namespace poly
}  // namespace zk

using namespace zk;
using namespace zk::poly;

static cudaError_t binary_op(PolyPtr r, ConstPolyPtr a, ConstPolyPtr b, u32 op, cudaStream_t stream) {
    u64 len = a.len < b.len ? a.len : b.len;
    u64 upper = a.len < b.len ? b.len : a.len;
    if (a.len < b.len) {
        std::swap(a, b);
        if (op == OP_SUB) op = OP_SUBR;
    }
    View vr, va, vb;
    ZK_CHECK_ARG(make_view(r, &vr) && make_view(a, &va) && make_view(b, &vb));
    ZK_CHECK_ARG(r.len >= upper);
    if (upper == 0) return cudaSuccess;
    binary_kernel<<<grid_for(upper, 256), 256, 0, stream>>>(vr, va, vb, len, upper, op);
    return cudaGetLastError();
}

extern "C" cudaError_t poly_add(PolyPtr r, ConstPolyPtr a, ConstPolyPtr b, cudaStream_t stream) {
    return binary_op(r, a, b, OP_ADD, stream);
}
extern "C" cudaError_t poly_sub(PolyPtr r, ConstPolyPtr a, ConstPolyPtr b, cudaStream_t stream) {
    return binary_op(r, a, b, OP_SUB, stream);
}
extern "C" cudaError_t poly_mul(PolyPtr r, ConstPolyPtr a, ConstPolyPtr b, cudaStream_t stream) {
    return binary_op(r, a, b, OP_MUL, stream);
}
extern "C" cudaError_t zkp_poly_square(PolyPtr r, ConstPolyPtr a, cudaStream_t stream) {
    return binary_op(r, a, a, OP_SQR, stream);
}

static cudaError_t fill(PolyPtr t, u32 kind, bool coef, cudaStream_t stream) {
    View v;
    ZK_CHECK_ARG(make_view(t, &v));
    if (v.len == 0) return cudaSuccess;
    fill_kernel<<<grid_for(v.len, 256), 256, 0, stream>>>(v, v.len, kind, coef);
    return cudaGetLastError();
}
extern "C" cudaError_t poly_one_lagrange(PolyPtr target, cudaStream_t stream) { return fill(target, 1, false, stream); }
extern "C" cudaError_t poly_one_coef(PolyPtr target, cudaStream_t stream) { return fill(target, 1, true, stream); }
extern "C" cudaError_t poly_zero(PolyPtr target, cudaStream_t stream) { return fill(target, 0, true, stream); }

extern "C" cudaError_t inv_scalar(unsigned int *target, cudaStream_t stream) {
    ZK_CHECK_ARG(target != nullptr);
    scalar_kernel<<<1, 32, 0, stream>>>(target, 0, 0);
    return cudaGetLastError();
}
extern "C" cudaError_t scalar_pow(unsigned int *target, unsigned long long exp, cudaStream_t stream) {
    ZK_CHECK_ARG(target != nullptr);
    scalar_kernel<<<1, 32, 0, stream>>>(target, exp, 1);
    return cudaGetLastError();
}

// ---- poly_eval: temp = CTA results and the next level's point, per level
extern "C" cudaError_t poly_eval(void *temp_buf, unsigned long *temp_buf_size, ConstPolyPtr poly, unsigned int *res,
                                 const unsigned int *x, cudaStream_t stream) {
    const u64 n = poly.len;
    const u32 c0 = chunk_for(n);
    const u64 m = ctas_for(n, c0);  // at most TOP_MAX: one CTA finishes
    const size_t need = al(m * 32) + (m > 1 ? al(32) : 0);
    if (temp_buf == nullptr) {
        ZK_CHECK_ARG(temp_buf_size != nullptr);
        *temp_buf_size = need;
        return cudaSuccess;
    }
    ZK_CHECK_ARG(res != nullptr && x != nullptr);
    if (temp_buf_size) ZK_CHECK_ARG(*temp_buf_size >= need);
    View v;
    ZK_CHECK_ARG(make_view(poly, &v));
    if (n == 0) return cudaMemsetAsync(res, 0, 32, stream);
    char *base = reinterpret_cast<char *>(temp_buf);
    u32 *part = reinterpret_cast<u32 *>(base), *point = reinterpret_cast<u32 *>(base + al(m * 32));
    eval_kernel<<<(u32)m, CTA, 0, stream>>>(v, n, x, c0, log2_of(c0), m == 1 ? res : part, m == 1 ? nullptr : point);
    ZK_TRY(cudaGetLastError());
    if (m == 1) return cudaSuccess;
    const u32 c1 = top_chunk(m);
    eval_kernel<<<1, CTA, 0, stream>>>(plain_view(part, m), m, point, c1, log2_of(c1), res, nullptr);
    return cudaGetLastError();
}

// ---- batched_invert: temp = running products, per-CTA products
extern "C" cudaError_t batched_invert(void *temp_buffer, unsigned long *buffer_size, PolyPtr poly,
                                      cudaStream_t stream) {
    const u64 n = poly.len;
    const u32 c = walk_chunk_for(n);
    const u64 m = ctas_for(n, c);
    const size_t need = al(n * 32) + 2 * al(m * 32);
    if (temp_buffer == nullptr) {
        ZK_CHECK_ARG(buffer_size != nullptr);
        *buffer_size = need;
        return cudaSuccess;
    }
    View v;
    ZK_CHECK_ARG(make_view(poly, &v));
    if (n == 0) return cudaSuccess;
    char *base = reinterpret_cast<char *>(temp_buffer);
    u32 *prefix = reinterpret_cast<u32 *>(base);
    u32 *tot = reinterpret_cast<u32 *>(base + al(n * 32));
    u32 *top_prefix = reinterpret_cast<u32 *>(base + al(n * 32) + al(m * 32));
    if (m == 1) {
        if (one_warp(n, c)) inv_one_kernel<true><<<1, 32, 0, stream>>>(v, (u32)n, c, prefix);
        else inv_one_kernel<false><<<1, CTA, 0, stream>>>(v, (u32)n, c, prefix);
        return cudaGetLastError();
    }
    inv_up_kernel<<<(u32)m, CTA, 0, stream>>>(v, n, c, prefix, tot);
    ZK_TRY(cudaGetLastError());
    inv_top_kernel<<<1, CTA, 0, stream>>>(tot, (u32)m, top_chunk(m), top_prefix);
    ZK_TRY(cudaGetLastError());
    inv_down_kernel<<<(u32)m, CTA, 0, stream>>>(v, n, c, prefix, tot);
    return cudaGetLastError();
}

// ---- scan_mul: inclusive product scan in place; temp = per-CTA products, and per-chunk ones where
// the chunks are of MAX_C elements or more
extern "C" cudaError_t scan_mul(void *temp_buffer, unsigned long *buffer_size, PolyPtr target, cudaStream_t stream) {
    const u64 n = target.len;
    const u32 c = walk_chunk_for(n);
    const u64 m = ctas_for(n, c);
    const size_t keep = c >= MAX_C ? al(m * CTA * 32) : 0;
    const size_t need = al(m * 32) + keep;
    if (temp_buffer == nullptr) {
        ZK_CHECK_ARG(buffer_size != nullptr);
        *buffer_size = need;
        return cudaSuccess;
    }
    View v;
    ZK_CHECK_ARG(make_view(target, &v));
    if (n == 0) return cudaSuccess;
    char *base = reinterpret_cast<char *>(temp_buffer);
    u32 *tot = reinterpret_cast<u32 *>(base), *ex = keep ? reinterpret_cast<u32 *>(base + al(m * 32)) : nullptr;
    if (m > 1) {
        scan_up_kernel<<<(u32)m, CTA, 0, stream>>>(v, n, c, ex, tot);
        ZK_TRY(cudaGetLastError());
        scan_top_kernel<<<1, CTA, 0, stream>>>(tot, (u32)m, top_chunk(m));
        ZK_TRY(cudaGetLastError());
    }
    if (one_warp(n, c)) scan_down_kernel<true><<<1, 32, 0, stream>>>(v, n, c, nullptr, nullptr);
    else scan_down_kernel<false><<<(u32)m, CTA, 0, stream>>>(v, n, c, ex, m > 1 ? tot : nullptr);
    return cudaGetLastError();
}

// ---- kate_division: q = (p - p(b)) / (X - b), length 2^log_p; temp = powers of b, CTA values, and
// chunk carries where the chunks are of MAX_C elements or more
extern "C" cudaError_t kate_division(void *temp_buf, unsigned long *temp_buf_size, unsigned int log_p, ConstPolyPtr p,
                                     const unsigned int *b, PolyPtr q, cudaStream_t stream) {
    const u64 n = 1ull << log_p;
    const u32 c = walk_chunk_for(n);
    const u64 m = ctas_for(n, c);
    const size_t keep = c >= MAX_C ? al(m * CTA * 32) : 0;
    const size_t need = m > 1 ? al(TAB * 32) + al(m * 32) + keep : 256;
    if (temp_buf == nullptr) {
        ZK_CHECK_ARG(temp_buf_size != nullptr);
        *temp_buf_size = need;
        return cudaSuccess;
    }
    ZK_CHECK_ARG(p.len == n && q.len == n && b != nullptr);
    View vp, vq;
    ZK_CHECK_ARG(make_view(p, &vp) && make_view(q, &vq));
    char *base = reinterpret_cast<char *>(temp_buf);
    u32 *tab = m > 1 ? reinterpret_cast<u32 *>(base) : nullptr;
    u32 *tot = reinterpret_cast<u32 *>(base + al(TAB * 32));
    u32 *carry = keep ? reinterpret_cast<u32 *>(base + al(TAB * 32) + al(m * 32)) : nullptr;
    if (m > 1) {
        kate_up_kernel<<<(u32)m, CTA, 0, stream>>>(vp, n, b, c, log2_of(c), carry, tot, tab);
        ZK_TRY(cudaGetLastError());
        const u32 c1 = top_chunk(m);
        kate_top_kernel<<<1, CTA, 0, stream>>>(tot, (u32)m, tab + (32 + WARPS) * 8, c1, log2_of(c1));
        ZK_TRY(cudaGetLastError());
    }
    if (one_warp(n, c))
        kate_down_kernel<true><<<1, 32, 0, stream>>>(vp, vq, n, b, c, log2_of(c), nullptr, nullptr, nullptr);
    else kate_down_kernel<false><<<(u32)m, CTA, 0, stream>>>(vp, vq, n, b, c, log2_of(c), carry, tot, tab);
    return cudaGetLastError();
}
#include "permute.cuh"
