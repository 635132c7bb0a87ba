// Radix-16 transform passes on the integer tensor cores (tcgen05.mma kind::i8).
//
// A 16-point DFT over Fr is a product with constants: X_k = sum_j x_j w16^(jk).  Written over
// the bytes of x_j (x_j = sum_i x_j[i] 2^(8i)) it is
//     X_k = sum_(j,i) x_j[i] * V(jk, i),   V(e, i) = w16^e 2^(8i) mod r,
// and over the bytes of the 32-byte constants V a plain matrix product of unsigned bytes with
// 32-bit sums: row = pencil, K index = (j, i), N index = (k, byte b).  Memory already holds
// the elements as bytes, so A is the data as it is.  The 32 column sums of an output are at most
// 8 * 32 * 255 * 255 < 2^24; adding them up with their weights 2^(8b) gives a value below 2^16 r
// (no reduction of a double-width product is needed), and one quotient digit brings it below 2r.
// What is left for the multiply pipe is one twiddle product an element per four index bits,
// where a radix-2 register pass needs two.
//
// The first radix-2 DIF stage is done in registers (s = x_j + x_(j+8), d = x_j - x_(j+8)), and
// the second for the even outputs, which leaves 8x8, 4x4 and 4x4 blocks of 32 x 32 bytes: 96 KB
// of constants, resident in shared memory for the whole (persistent) launch.  A CTA runs three
// independent groups of 128 threads; a group owns one tile of 128 pencils (one per thread and
// per TMEM lane), 32 KB of A and 128 TMEM columns (four outputs), so while one group waits for its
// products the other two read theirs and multiply by twiddles.
//
// Measured at 2^24: 0.44 ms a pass (the first, whose roots come from DRAM, 0.51) for four bits, where
// the register pass takes 0.70 for five; the whole transform 3.39 -> 2.84 ms.  At 2^22 the multiply
// pipe is 62 % busy, the tensor pipe 10 %, DRAM 26 %: what bounds it is the latency of each warp's
// chain with three warps a scheduler.  Four groups need 128 registers a thread and spill (3.43 ms);
// keeping the even half's sums in memory instead of registers avoids that but costs more (3.31 ms
// with four groups, 3.27 with three); lanes over 32 neighbouring pencils, each with a twiddle of its
// own, 3.51 ms.
#pragma once
#include "common.cuh"

namespace zk {
namespace ntt {

constexpr u32 UM_D = 4;                        // index bits per pass
constexpr u32 UM_GROUPS = 3;                   // tiles in flight per CTA
constexpr u32 UM_ROWS = 128;                   // pencils per tile (MMA M)
constexpr u32 UM_COLS = 128;                   // TMEM columns per group (MMA N)
constexpr u32 UM_B_SD = 256 * 256;             // offsets of the constant blocks
constexpr u32 UM_B_SS = UM_B_SD + 128 * 128;
constexpr u32 UM_A = UM_B_SS + 128 * 128;      // the groups' A tiles
constexpr u32 UM_A_BYTES = UM_ROWS * 256;
constexpr u32 UM_BAR = UM_A + UM_GROUPS * UM_A_BYTES;  // one mbarrier a group, then the TMEM address
constexpr u32 UM_SMEM = UM_BAR + 64;
// D = S32, A and B unsigned bytes, both K-major, N = 128, M = 128
constexpr u32 UM_IDESC = (2u << 4) | ((UM_COLS >> 3) << 17) | ((UM_ROWS >> 4) << 24);
// A wait for the tensor core (some microseconds) gives up after a second, and whatever the clock says
// after UM_POLLS polls of an mbarrier.  Its group then stores nothing more, waits once more for what is
// in flight, sets the context's status word (zkp_ntt_status) and leaves.
constexpr u32 UM_WAIT_NS = 1000000000u, UM_POLLS = 1u << 24;

ZK_DI u32 um_smem_addr(const void *p) { return (u32)__cvta_generic_to_shared(p); }
// shared-memory matrix descriptor: no swizzle, K-major; core matrices of 8 rows x 16 bytes,
// 128 bytes apart along M / N, `lbo` bytes apart along K
ZK_DI u64 um_desc(u32 addr, u32 lbo) {
    return (u64)((addr >> 4) & 0x3fffu) | ((u64)(lbo >> 4) << 16) | ((u64)(128u >> 4) << 32) | (1ull << 46);
}
ZK_DI void um_mma(u32 tmem, u64 a, u64 b, bool accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::i8 [%0], %1, %2, %3, p;\n\t}\n" ::"r"(tmem),
        "l"(a), "l"(b), "r"(UM_IDESC), "r"(accumulate ? 1u : 0u)
        : "memory");
}
ZK_DI void um_commit(u32 bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar) : "memory");
}
ZK_DI u64 um_clock_ns() {
    u64 t;
    asm volatile("mov.u64 %0, %globaltimer;" : "=l"(t));
    return t;
}
// limit 0: gives up at once
ZK_DI bool um_wait(u32 bar, u32 parity, u32 limit_ns) {
    u64 start = 0;
    for (u32 i = 0; limit_ns && i < UM_POLLS; i++) {
        u32 done;
        asm volatile(
            "{\n\t.reg .pred p;\n\t"
            "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
            "selp.b32 %0, 1, 0, p;\n\t}\n"
            : "=r"(done)
            : "r"(bar), "r"(parity)
            : "memory");
        if (done) return true;
        const u64 now = um_clock_ns();
        if (i == 0) start = now;
        if (now - start >= limit_ns) break;
    }
    return false;
}
ZK_DI void um_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
ZK_DI void um_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
ZK_DI void um_fence_async() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }
// group barrier; whether any thread of the group passed true
ZK_DI bool um_group_any(u32 g, bool f) {
    u32 any;
    asm volatile(
        "{\n\t.reg .pred p, q;\n\t"
        "setp.ne.u32 p, %2, 0;\n\t"
        "bar.red.or.pred q, %1, 128, p;\n\t"
        "selp.u32 %0, 1, 0, q;\n\t}\n"
        : "=r"(any)
        : "r"(g + 1), "r"(f ? 1u : 0u)
        : "memory");
    return any != 0;
}

// the warp's 32 TMEM lanes x 32 columns: this thread's row
ZK_DI void um_load32(u32 tmem, u32 *c) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
        "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16, %17, %18, %19, %20, %21, %22, "
        "%23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];\n\t"
        "tcgen05.wait::ld.sync.aligned;"
        : "=r"(c[0]), "=r"(c[1]), "=r"(c[2]), "=r"(c[3]), "=r"(c[4]), "=r"(c[5]), "=r"(c[6]), "=r"(c[7]), "=r"(c[8]),
          "=r"(c[9]), "=r"(c[10]), "=r"(c[11]), "=r"(c[12]), "=r"(c[13]), "=r"(c[14]), "=r"(c[15]), "=r"(c[16]),
          "=r"(c[17]), "=r"(c[18]), "=r"(c[19]), "=r"(c[20]), "=r"(c[21]), "=r"(c[22]), "=r"(c[23]), "=r"(c[24]),
          "=r"(c[25]), "=r"(c[26]), "=r"(c[27]), "=r"(c[28]), "=r"(c[29]), "=r"(c[30]), "=r"(c[31])
        : "r"(tmem)
        : "memory");
}

// 32-byte global accesses (32-byte aligned)
ZK_DI Fr um_ld(const u32 *p) {
    Fr r;
    asm volatile("ld.global.v8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                 : "=r"(r.v[0]), "=r"(r.v[1]), "=r"(r.v[2]), "=r"(r.v[3]), "=r"(r.v[4]), "=r"(r.v[5]), "=r"(r.v[6]),
                   "=r"(r.v[7])
                 : "l"(p)
                 : "memory");
    return r;
}
ZK_DI Fr um_ld_nc(const u32 *p) {
    Fr r;
    asm("ld.global.nc.v8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
        : "=r"(r.v[0]), "=r"(r.v[1]), "=r"(r.v[2]), "=r"(r.v[3]), "=r"(r.v[4]), "=r"(r.v[5]), "=r"(r.v[6]), "=r"(r.v[7])
        : "l"(p));
    return r;
}
ZK_DI void um_st(u32 *p, const Fr &x) {
    asm volatile("st.global.v8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"l"(p), "r"(x.v[0]), "r"(x.v[1]),
                 "r"(x.v[2]), "r"(x.v[3]), "r"(x.v[4]), "r"(x.v[5]), "r"(x.v[6]), "r"(x.v[7])
                 : "memory");
}

// a + b and a - b + 2m without a fold: at most 4m for a, b <= 2m, so still 256 bits
ZK_DI Fr um_add_raw(const Fr &a, const Fr &b) {
    Fr r;
    r.v[0] = add_cc(a.v[0], b.v[0]);
#pragma unroll
    for (int i = 1; i < 7; i++) r.v[i] = addc_cc(a.v[i], b.v[i]);
    r.v[7] = addc(a.v[7], b.v[7]);
    return r;
}
ZK_DI Fr um_sub_raw(const Fr &a, const Fr &b) {
    Fr r;
    r.v[0] = add_cc(a.v[0], FrParams::m2(0));
#pragma unroll
    for (int i = 1; i < 7; i++) r.v[i] = addc_cc(a.v[i], FrParams::m2(i));
    r.v[7] = addc(a.v[7], FrParams::m2(7));
    Fr::sub_raw(r.v, r.v, b.v);
    return r;
}

// element j of the thread's row into the A tile: two 16-byte chunks of K
ZK_DI void um_put(unsigned char *A, u32 j, u32 row, const Fr &x) {
    *reinterpret_cast<uint4 *>(A + (2 * j) * (UM_ROWS * 16) + row * 16) = make_uint4(x.v[0], x.v[1], x.v[2], x.v[3]);
    *reinterpret_cast<uint4 *>(A + (2 * j + 1) * (UM_ROWS * 16) + row * 16) = make_uint4(x.v[4], x.v[5], x.v[6], x.v[7]);
}

// sum_b c_b 2^(8b) mod r in [0, 2r) for column sums c_b <= 8 * 32 * 255^2: pairs of columns
// still fit a word (c_b + 256 c_(b+1) < 2^32), the sixteen pairs are added at 16-bit spacing, and
// the quotient digit floor((T / 2^240) floor(2^285 / r) / 2^45) is floor(T / r) or one less
ZK_DI Fr um_combine(const u32 *c) {
    u32 p[16];
#pragma unroll
    for (int i = 0; i < 16; i++) p[i] = c[2 * i] + (c[2 * i + 1] << 8);
    Fr t;
    t.v[0] = p[0];
    t.v[1] = add_cc(p[2], p[1] >> 16);
#pragma unroll
    for (int i = 2; i < 8; i++) t.v[i] = addc_cc(p[2 * i], p[2 * i - 1] >> 16);
    u32 t8 = addc(p[15] >> 16, 0u);
    t.v[0] = add_cc(t.v[0], p[1] << 16);
#pragma unroll
    for (int i = 1; i < 8; i++) t.v[i] = addc_cc(t.v[i], p[2 * i + 1] << 16);
    t8 = addc(t8, 0u);
    const u32 q = __umulhi((t8 << 16) | (t.v[7] >> 16), 0xa948e8c4u) >> 13;  // floor(2^285 / r)
    t.v[0] = mad_lo_cc(q, FrParams::np(0), t.v[0]);
    t.v[1] = madc_hi_cc(q, FrParams::np(0), t.v[1]);
    t.v[2] = madc_lo_cc(q, FrParams::np(2), t.v[2]);
    t.v[3] = madc_hi_cc(q, FrParams::np(2), t.v[3]);
    t.v[4] = madc_lo_cc(q, FrParams::np(4), t.v[4]);
    t.v[5] = madc_hi_cc(q, FrParams::np(4), t.v[5]);
    t.v[6] = madc_lo_cc(q, FrParams::np(6), t.v[6]);
    t.v[7] = madc_hi(q, FrParams::np(6), t.v[7]);
    t.v[1] = mad_lo_cc(q, FrParams::np(1), t.v[1]);
    t.v[2] = madc_hi_cc(q, FrParams::np(1), t.v[2]);
    t.v[3] = madc_lo_cc(q, FrParams::np(3), t.v[3]);
    t.v[4] = madc_hi_cc(q, FrParams::np(3), t.v[4]);
    t.v[5] = madc_lo_cc(q, FrParams::np(5), t.v[5]);
    t.v[6] = madc_hi_cc(q, FrParams::np(5), t.v[6]);
    t.v[7] = madc_lo_cc(q, FrParams::np(7), t.v[7]);
    return t;
}

// The thread's pencil in tile `item` (row = its row): lower index bits c and upper bits h, of
// log_h bits.  Lanes take 4 neighbouring c and 8 h where there are that many: a 128-byte line of data
// is read by four lanes, and a warp needs only four different twiddles an output, where 32
// neighbouring c would need 32.
ZK_DI void um_pencil(u64 item, u32 row, u32 lo, u32 log_h, u64 &c, u64 &h) {
    const u32 hb = log_h < 5 ? log_h : 5, cb = 7 - hb;  // row bits of h and c: c's low two come first
    h = ((item >> (lo - cb)) << hb) | ((row >> 2) & ((1u << hb) - 1));
    c = ((item & ((1ull << (lo - cb)) - 1)) << cb) | ((row >> (2 + hb)) << 2) | (row & 3);
}

// The twiddle product is the Montgomery one also for callers with a Shoup table: these passes wait
// for loads more than for the multiply pipe, and its root is 32 bytes, not 64 (2^24 2.92 -> 2.83 ms,
// 2^22 0.752 -> 0.738).
__global__ void __launch_bounds__(UM_GROUPS * 128, 1) ntt_umma_kernel(const PassArgs a, u32 items, u32 limit_ns,
                                                                       u32 *status) {
    extern __shared__ __align__(1024) unsigned char um_sm[];
    const u32 tid = threadIdx.x, g = tid >> 7, row = tid & 127;
    const u32 L = a.L, lo = a.lo;
    u32 *slot = reinterpret_cast<u32 *>(um_sm + UM_BAR + 8 * UM_GROUPS);
    const u32 bar = um_smem_addr(um_sm + UM_BAR) + 8 * g;

    if (tid < 32) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], 512;" ::"r"(um_smem_addr(slot))
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
    }
    if (row == 0) {
        asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(bar) : "memory");
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    // ---- the constants: V(e, i) as bytes [e][i / 16][b][i % 16] in the A area, then copied to the
    // places (n, k) of the three blocks that use them
    unsigned char *U = um_sm + UM_A;
    for (u32 v = tid; v < 512; v += UM_GROUPS * 128) {
        const u32 e = v >> 5, i = v & 31;
        Fr p2 = Fr::zero();
#pragma unroll
        for (u32 w = 0; w < 8; w++) p2.v[w] = w == (i >> 2) ? 1u << (8 * (i & 3)) : 0u;
        Fr x = Fr::mul(table_root(a.tw, (u64)e << (L - UM_D), L), p2);
        x = x.canonical();
        unsigned char *dst = U + e * 1024 + (i >> 4) * 512 + (i & 15);
#pragma unroll
        for (u32 b = 0; b < 32; b++) dst[b * 16] = (unsigned char)(x.v[b >> 2] >> (8 * (b & 3)));
    }
    __syncthreads();
    for (u32 v = tid; v < 6144; v += UM_GROUPS * 128) {
        const u32 blk = v < 4096 ? 0 : (v < 5120 ? 1 : 2);
        const u32 x = blk == 0 ? v : (v - 4096) & 1023;
        const u32 kc = blk == 0 ? x >> 8 : x >> 7, n = blk == 0 ? x & 255 : x & 127;
        const u32 o = n >> 5, b = n & 31, j = kc >> 1, ih = kc & 1;
        const u32 e = (blk == 0 ? j * (2 * o + 1) : blk == 1 ? 2 * j * (2 * o + 1) : 4 * j * o) & 15;
        const u32 off = blk == 0 ? kc * 4096 + n * 16 : (blk == 1 ? UM_B_SD : UM_B_SS) + kc * 2048 + n * 16;
        *reinterpret_cast<uint4 *>(um_sm + off) = *reinterpret_cast<const uint4 *>(U + e * 1024 + ih * 512 + b * 16);
    }
    um_fence_async();
    um_fence_before();
    __syncthreads();
    um_fence_after();
    const u32 tmem = *slot + g * UM_COLS;
    const u32 tmem_row = tmem + (((tid >> 5) & 3) << 21);  // lanes 32 w .. of warp w of the group
    unsigned char *A = um_sm + UM_A + g * UM_A_BYTES;
    const u32 a_addr = um_smem_addr(A), b_addr = um_smem_addr(um_sm);
    u32 parity = 0;
    bool late = false;  // a wait of this warp ran out

    // `steps` K steps of 32 bytes from A offset a_off and the constant block at b_off; false, and nothing
    // issued, once a wait of the group has run out
    auto issue = [&](u32 a_off, u32 b_off, u32 b_lbo, u32 steps) {
        um_fence_before();
        if (um_group_any(g, late)) return false;
        if (row == 0) {
            um_fence_after();
            for (u32 s = 0; s < steps; s++)
                um_mma(tmem, um_desc(a_addr + a_off + s * 2 * (UM_ROWS * 16), UM_ROWS * 16),
                       um_desc(b_addr + b_off + s * 2 * b_lbo, b_lbo), s > 0);
            um_commit(bar);
        }
        return true;
    };
    auto finish = [&]() {
        if (!um_wait(bar, parity, limit_ns)) {
            late = true;
            um_wait(bar, parity, UM_WAIT_NS);  // still in flight: reads A, writes TMEM
        }
        late = __any_sync(0xffffffffu, late);
        parity ^= 1;
        um_fence_after();
    };

    u64 base = 0, c = 0;
    const u64 half = 1ull << (L - 1);
    const u32 esh = L - lo - UM_D;
    auto root = [&](u32 k) { return um_ld_nc(a.tw + (((c * k) << esh) & (half - 1)) * 8); };
    // outputs k = k0, k0 + dk, ... (four of them) from the group's TMEM columns; an output's twiddle
    // is loaded one output ahead
    auto drain = [&](u32 k0, u32 dk, Fr r) {
        if (late) return;
#pragma unroll 1
        for (u32 o = 0; o < 4; o++) {
            const u32 k = k0 + o * dk;
            u32 cs[32];
            um_load32(tmem_row + o * 32, cs);
            const Fr next = root(k + dk);  // past the last one: in range, unused
            Fr x = um_combine(cs);
            if (k != 0) {
                x = Fr::mul(x, r);
                // w^(n/2) = -1.  2r - 0 is 2r itself: these passes store and take the closed range [0, 2r]
                // (a sum of two is at most 4r and folds to at most 2r).  The last pass, in registers,
                // canonicalises [0, 2r) only, and meets no more: its outputs are a + b and a - b with a the
                // first element of a butterfly block, which is the pencil's element 0 plus and minus
                // others, never multiplied.  That one came from c = 0, is not flipped and so below 2r,
                // and a +- b folded is below 2r if a is and b is at most 2r.
                if (((c * k) << esh) >= half) {
                    Fr m2;
#pragma unroll
                    for (int i = 0; i < 8; i++) m2.v[i] = FrParams::m2(i);
                    Fr::sub_raw(x.v, m2.v, x.v);
                }
            }
            um_st(a.v.at(base + ((u64)(__brev(k) >> 28) << lo)), x);
            r = next;
        }
    };

    for (u64 item = blockIdx.x + (u64)gridDim.x * g; item < items; item += (u64)gridDim.x * UM_GROUPS) {
        u64 h;
        um_pencil(item, row, lo, esh, c, h);
        base = (h << (lo + UM_D)) | c;
        Fr s[8];
#pragma unroll
        for (u32 j = 0; j < 8; j++) {
            const Fr x0 = um_ld(a.v.at(base + ((u64)j << lo)));
            const Fr x1 = um_ld(a.v.at(base + ((u64)(j + 8) << lo)));
            s[j] = Fr::add(x0, x1);
            um_put(A, j, row, um_sub_raw(x0, x1));
        }
        um_fence_async();
        if (!issue(0, 0, 4096, 8)) break;  // outputs 1, 3, 5, 7
        Fr r = root(1);
        finish();
        drain(1, 2, r);
        if (!issue(0, 128 * 16, 4096, 8)) break;  // outputs 9, 11, 13, 15
        r = root(9);
        finish();
        // A is free again: the even half's second stage
#pragma unroll
        for (u32 j = 0; j < 4; j++) {
            um_put(A, j, row, um_add_raw(s[j], s[j + 4]));
            um_put(A, j + 4, row, um_sub_raw(s[j], s[j + 4]));
        }
        um_fence_async();
        drain(9, 2, r);
        if (!issue(4 * 2 * (UM_ROWS * 16), UM_B_SD, 2048, 4)) break;  // outputs 2, 6, 10, 14
        r = root(2);
        finish();
        drain(2, 4, r);
        if (!issue(0, UM_B_SS, 2048, 4)) break;  // outputs 0, 4, 8, 12
        finish();
        drain(0, 4, r);
    }
    if (late && (tid & 31) == 0) {
        *(volatile u32 *)status = 1;
        __threadfence_system();
    }
    um_fence_before();
    __syncthreads();
    if (tid < 32)
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, 512;" ::"r"(*slot));
}

}  // namespace ntt
}  // namespace zk
