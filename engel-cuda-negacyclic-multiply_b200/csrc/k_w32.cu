// Kernels of the 30-bit word engine (w32.cuh): k_dec_tc32 (residues on the tensor cores + forward
// column stages), k_row32 (row blocks) and k_crt_tc32 (inverse column stages + CRT on the tensor
// cores), with their launchers.
//
// Residues. With x_n given as 4 L bytes x_{n,b}, x_n mod p_i = sum_c 2^(8 c) S[n][i,c] with
// S[n][i,c] = sum_b x_{n,b} w_{i,b,c}, w_{i,b,c} byte c (of 4) of 2^(8 b) mod p_i: the same u8 x u8
// contraction as the 62-bit engine's k_dec_tc, with four byte planes a prime instead of eight, so
// one pass of MMAs (128 accumulator columns) covers 32 primes. The four sums are folded and reduced
// together (fold_planes).
//
// CRT. The 4 bytes of each residue against a per-plan table (K = 4 k <= 256 bytes) that carries the
// factors y_i, the reduction of M/p_i mod q and the quotient (below, at the CRT's kernels).
#include "batch_types.h"
#include "crt_tc.cuh"
#include "kernel_registry.h"
#include "w32.cuh"

namespace nc {

namespace w32 {

namespace {

using crt_tc_detail::kmajor_desc;
using crt_tc_detail::smem_u32;

__device__ __forceinline__ void cp_async16(void* dst, const void* src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_u32(dst)), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async8(void* dst, const void* src, uint32_t src_bytes) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;" ::"r"(smem_u32(dst)), "l"(src), "r"(src_bytes)
                 : "memory");
}
__device__ __forceinline__ void cp_async4(void* dst, const void* src, uint32_t src_bytes) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(smem_u32(dst)), "l"(src), "r"(src_bytes)
                 : "memory");
}
// One thread: `bytes` (a multiple of 16) to shared memory by a bulk copy that completes phase 0 of `bar`.
__device__ __forceinline__ void bulk_table(void* dst, const void* src, uint32_t bytes, uint32_t bar) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                     smem_u32(dst)),
                 "l"(src), "r"(bytes), "r"(bar)
                 : "memory");
}
__device__ __forceinline__ uint64_t mad_wide(uint32_t a, uint32_t b, uint64_t c) {
    uint64_t d;
    asm("mad.wide.u32 %0, %1, %2, %3;" : "=l"(d) : "r"(a), "r"(b), "l"(c));
    return d;
}

// sum_c 2^(8 c) s[c] mod p into [0, 3.9 p) (the butterflies take [0, 4p)), for s[c] < 2^23 and p in
// (7/8 2^30, 2^30): with lo = s0 + 2^8 s1 and hi = s2 + 2^8 s3 (both below 2^31.01), V = lo + 2^16 hi and
// q = floor(hi floor(2^48 / p) / 2^32) falls short of 2^16 hi / p by less than 1 + hi / 2^32 < 1.6, and
// lo < 2.3 p is not reduced: V - q p < 3.9 p. Five instructions, one of them a multiply-high (a 48-bit
// sum and its Barrett quotient took ten).
__device__ __forceinline__ uint32_t fold_planes(const uint32_t* s, uint32_t p, uint32_t c48) {
    const uint32_t lo = s[0] + (s[1] << 8), hi = s[2] + (s[3] << 8);
    return lo + (hi << 16) - __umulhi(hi, c48) * p;
}

// Residue row of prime il of the pass group (128 u32) over its pair's 1 KB of weights.
__device__ __forceinline__ uint32_t* res_row(uint8_t* sB, int il) { return reinterpret_cast<uint32_t*>(sB + il * 512); }

// Slot of tile row x in prime i's residue row. Every prime's row starts on bank 0, so rows are
// XORed (bits 2-4 for 4-column tiles, bits 0-4 otherwise) by the prime and, for 4-column tiles,
// by the half of the 32-point column (bit 5): the column stages' loads of one warp then fall on
// 32 different banks, and the fold's stores (32 consecutive rows) stay conflict-free.
__device__ __forceinline__ int res_slot(int i, int x, int C) {
    const int f = C == 4 ? ((((i & 3) << 1) | ((x >> 5) & 1)) << 2) : ((i * C) & 31);
    return x ^ f;
}

// Weight pairs a launch copies: the primes rounded up to a multiple of four (an MMA's N is a
// multiple of 16 columns), within the table's 64 primes.
__host__ __device__ constexpr int dec32_weight_pairs(int k) { return ((k + 3) & ~3) / 2; }

// Neighbouring columns a thread of the column stages takes (VJ): sixteen values in registers. Thirty-two
// spill at 64 registers and leave threads idle (64 x 16384, 8-point columns: 946, 897 and 983 us a batch
// with one, two and four columns; N = 65536, 16-point columns: 74.9 and 76.1 us a product with one and two).
__host__ __device__ constexpr int column_width(int logN1) { return logN1 <= 2 ? 4 : logN1 == 3 ? 2 : 1; }

// Forward column stages of one prime: 2^LOG_N1 points of each of the tile's columns.
template <int LOG_N1, int CC, int LN2>
__device__ __forceinline__ void dec32_columns(uint32_t* R, const uint2* tw0, const uint2* s_pc, uint8_t* sB, int N,
                                              int N2, int logC, int j0, int i0, int i1) {
    constexpr int N1 = 1 << LOG_N1;
    const int C = CC ? CC : 1 << logC;
    const int tid = int(threadIdx.x), lane = tid & 31;
    if constexpr (LOG_N1 == 5) {
        // 32-point columns on two adjacent lanes, as in k_dec_tc: lane h runs the first stage's
        // butterflies (u, u + 16) for u in [8h, 8h + 8), the lanes swap halves, and each runs the
        // four remaining stages on its half-subtree (twiddle root 2 + h)
        const int total = 2 * (i1 - i0) * C;
        for (int w0 = tid & ~31; w0 < total; w0 += kThreads) {
            const int w = w0 + lane;
            const bool active = w < total;
            const int item = active ? w >> 1 : 0, h = w & 1;
            const int i = i0 + (item >> logC), j = item & (C - 1);
            const uint32_t* sr = res_row(sB, i - i0);
            const uint32_t p = s_pc[i - i0].x, p2 = 2 * p;
            const uint2* tw = tw0 + size_t(i) * kMaxN;
            uint32_t xs[8], ys[8];
            const uint2 w1 = __ldg(tw + 1);
#pragma unroll
            for (int e = 0; e < 8; ++e) {
                const int u = 8 * h + e;
                xs[e] = sr[res_slot(i, u * C + j, C)];
                ys[e] = sr[res_slot(i, (u + 16) * C + j, C)];
                w32::ct_bfly(xs[e], ys[e], w1.x, w1.y, p, p2);
            }
            uint32_t v[1][16];
#pragma unroll
            for (int e = 0; e < 8; ++e) {
                const uint32_t got = __shfl_xor_sync(0xffffffffu, h ? xs[e] : ys[e], 1);
                v[0][e] = h ? got : xs[e];
                v[0][8 + e] = h ? ys[e] : got;
            }
            w32::column_forward_root<4, 1>(tw, 2 + h, p, v);
            if (active) {
                uint32_t* out = R + size_t(i) * N + j0 + j + size_t(16 * h) * N2;
#pragma unroll
                for (int u = 0; u < 16; ++u) __stcg(out + size_t(u) * N2, v[0][u]);
            }
        }
    } else if constexpr (CC > 0) {
        // VJ neighbouring columns of a prime a thread: 16- or 8-byte shared loads and stores, and one set
        // of twiddles and addresses for all of them. Rows u C + j
        // XORed by (i C) mod 32 are (u ^ (i mod 32 / C)) C + j.
        constexpr int VJ = column_width(LOG_N1), GP = CC / VJ;
        constexpr int X = CC < 32 ? 32 / CC : 1;
        const int total = (i1 - i0) * GP;
#pragma unroll 1
        for (int w = tid; w < total; w += kThreads) {
            const int il = w / GP, j = (w % GP) * VJ;
            const int x = il & (X - 1);  // i0 is a multiple of 32
            const uint32_t* sr = res_row(sB, il) + j;
            const uint32_t p = s_pc[il].x;
            uint32_t v[VJ][N1];
#pragma unroll
            for (int u = 0; u < N1; ++u) {
                const uint32_t* at = sr + ((u & ~(X - 1)) + ((u & (X - 1)) ^ x)) * CC;
                if constexpr (VJ == 4) {
                    const uint4 q = *reinterpret_cast<const uint4*>(at);
                    v[0][u] = q.x;
                    v[1][u] = q.y;
                    v[2][u] = q.z;
                    v[3][u] = q.w;
                } else if constexpr (VJ == 2) {
                    const uint2 q = *reinterpret_cast<const uint2*>(at);
                    v[0][u] = q.x;
                    v[1][u] = q.y;
                } else {
                    v[0][u] = *at;
                }
            }
            if (LOG_N1 > 0) w32::column_forward_root<LOG_N1, VJ>(tw0 + size_t(i0 + il) * kMaxN, 1, p, v);
            uint32_t* out = R + size_t(i0 + il) * N + j0 + j;
#pragma unroll
            for (int u = 0; u < N1; ++u) {
                if constexpr (VJ == 4)
                    __stcg(reinterpret_cast<uint4*>(out + size_t(u) * N2), make_uint4(v[0][u], v[1][u], v[2][u], v[3][u]));
                else if constexpr (VJ == 2)
                    __stcg(reinterpret_cast<uint2*>(out + size_t(u) * N2), make_uint2(v[0][u], v[1][u]));
                else
                    __stcg(out + size_t(u) * N2, v[0][u]);
            }
        }
    } else {
        const int total = (i1 - i0) << logC;
#pragma unroll 1
        for (int w = tid; w < total; w += kThreads) {
            const int i = i0 + (w >> logC), j = w & (C - 1);
            const uint32_t* sr = res_row(sB, i - i0);
            uint32_t v[1][N1];
#pragma unroll
            for (int u = 0; u < N1; ++u) v[0][u] = sr[res_slot(i, u * C + j, C)];
            if (LOG_N1 > 0) w32::column_forward_root<LOG_N1, 1>(tw0 + size_t(i) * kMaxN, 1, s_pc[i - i0].x, v);
            uint32_t* out = R + size_t(i) * N + j0 + j;
#pragma unroll
            for (int u = 0; u < N1; ++u) __stcg(out + size_t(u) * N2, v[0][u]);
        }
    }
}

// CC: the tile's columns when N >= 128 (128 >> LOG_N1, a constant: the index arithmetic of the
// fold and the column stages folds away), 0 for smaller N. LN2: log2 N2 where it is 12 (the stores'
// offsets are then constants), else 0. Primes [i0, i1), i0 a multiple of 32.
template <int LOG_N1, int CC, int LN2>
__device__ __forceinline__ void dec_tc32_item(const ProductDesc& d, const Tables& t, int operand, int tile, int i0,
                                              int i1, bool early, uint8_t* smem, uint64_t (&bars)[2],
                                              uint32_t& taddr_slot) {
    uint64_t& bar = bars[0];
    const int N = 1 << d.logN;
    const int N2 = LN2 ? 1 << LN2 : N >> LOG_N1;
    const int T = CC ? kDecTcRows : (N < kDecTcRows ? N : kDecTcRows);
    const int logC = CC ? 7 - LOG_N1 : (N < kDecTcRows ? int(d.logN) : 7) - LOG_N1;
    const int C = CC ? CC : 1 << logC;
    const int j0 = tile * C;
    const int L = int(d.L), k = i1 - i0;
    const int wpairs = dec32_weight_pairs(k);
    const uint32_t* x = factor_limbs(d, operand);
    uint32_t* R = reinterpret_cast<uint32_t*>(factor_residues(d, operand));
    uint8_t* sA = smem;                     // [16 row groups][8 K chunks][8 rows][16 B]
    uint8_t* sB = smem + kDecTcRows * 128;  // [prime pair][8 K chunks][8 rows][16 B]
    uint2* s_pc = reinterpret_cast<uint2*>(sB + wpairs * 1024);  // p, floor(2^48 / p)
    const int tid = int(threadIdx.x), warp = tid >> 5, lane = tid & 31;

    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&taddr_slot)),
                     "r"(kDecTcCols)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    if (tid == 0) {
        asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_u32(&bar)) : "memory");
        asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_u32(&bars[1])) : "memory");
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        // the weights, already in shared-memory order, as one copy that the thread of the MMAs waits for
        bulk_table(sB, t.res_w32 + size_t(i0 >> 1) * 64, uint32_t(wpairs) * 1024u, smem_u32(&bars[1]));
    }
    __syncthreads();

    for (int w = tid; w < 2 * wpairs; w += kThreads) {
        const PrimeConst32 pc = t.pc32[i0 + w];  // the MMAs' primes
        s_pc[w] = make_uint2(pc.p, pc.c48);
    }
    if (early) pdl_trigger();
    pdl_wait();  // the operand and the residue rows belong to the stream's previous kernels
    // after the wait (and with the CTA's tensor memory in hand): the next kernel's CTAs are then placed
    // beside running CTAs, not beside a queue of waiting ones; at the kernel's entry, products of
    // N = 4096 to 16384 had kernels of two products resident at once, several row CTAs stacked on one
    // SM (N = 8192, 868 bits: 28.7 us a product, 20.3 us with the trigger here); where early_triggers
    // says so, before the wait
    pdl_trigger();
    const int kbytes = 4 * L;
    for (int q = tid; q < kDecTcRows * 8; q += kThreads) {
        const int rlo = q & 7, kc = (q >> 3) & 7, rg = q >> 6;
        const int m = rg * 8 + rlo;
        uint8_t* dst = sA + rg * 1024 + kc * 128 + rlo * 16;
        if (m < T && kc * 16 < kbytes) {
            const int n = (m >> logC) * N2 + j0 + (m & (C - 1));
            const uint32_t* row = x + size_t(n) * size_t(L);
            const int l0 = kc * 4;
            if ((L & 3) == 0) {
                cp_async16(dst, row + l0);
            } else if ((L & 1) == 0) {
                cp_async8(dst, row + l0, 8u);
                cp_async8(dst + 8, l0 + 2 < L ? row + l0 + 2 : row, l0 + 2 < L ? 8u : 0u);
            } else {
#pragma unroll
                for (int w = 0; w < 4; ++w) cp_async4(dst + 4 * w, l0 + w < L ? row + l0 + w : row, l0 + w < L ? 4u : 0u);
            }
        } else {
            *reinterpret_cast<uint4*>(dst) = make_uint4(0u, 0u, 0u, 0u);
        }
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    // (the thread of the MMAs has also waited for the weights)
    bool ok = __syncthreads_and(tid != 0 || bar_wait(t, smem_u32(&bars[1]), 0, kGiveUpCopies) ? 1 : 0) != 0;
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t taddr = taddr_slot;
    const int slices = (kbytes + 31) / 32;

    // passes of 32 primes; warp w reads tensor-memory lanes 32 (w % 4) .. and half w / 4 of the
    // pass's primes (16 of them, four per 16-column load)
    const int m = 32 * (warp & 3) + lane;
    const int half = warp >> 2;
    // a prime's place in its residue row depends on the prime mod 4 only (CC a constant)
    int slot[4];
#pragma unroll
    for (int e = 0; e < 4; ++e) slot[e] = CC ? res_slot(e, m, CC) : 0;
    for (int g = 0; ok && g * kDecTc32PassPrimes < k; ++g) {
        const int ig = g * kDecTc32PassPrimes;
        const int np = k - ig < kDecTc32PassPrimes ? k - ig : kDecTc32PassPrimes;
        if (tid == 0) {
            const uint32_t ncols = uint32_t(((np + 3) & ~3) * 4);
            const uint32_t idesc = (2u << 4) | ((ncols >> 3) << 17) | (uint32_t(kDecTcRows >> 4) << 24);
            const uint32_t a0 = smem_u32(sA), b0 = smem_u32(sB + (ig >> 1) * 1024);
            for (int s = 0; s < slices; ++s) {
                const uint64_t da = kmajor_desc(a0 + uint32_t(s) * 256u, 128u, 1024u);
                const uint64_t db = kmajor_desc(b0 + uint32_t(s) * 256u, 128u, 1024u);
                asm volatile(
                    "{\n\t.reg .pred p;\n\t"
                    "setp.ne.b32 p, %4, 0;\n\t"
                    "tcgen05.mma.cta_group::1.kind::i8 [%0], %1, %2, %3, p;\n\t}" ::"r"(taddr),
                    "l"(da), "l"(db), "r"(idesc), "r"(s));
            }
            asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(
                             smem_u32(&bar))
                         : "memory");
        }
        // one warp polls, the others wait at the barrier (eight polling warps took an eighth of the issue slots)
        ok = __syncthreads_and(warp != 0 || bar_wait(t, smem_u32(&bar), uint32_t(g & 1), kGiveUpMmas) ? 1 : 0) != 0;
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        const int ib = ig + 16 * half;
        const int ie = ig + np < ib + 16 ? ig + np : ib + 16;
        if (ok) {
            const uint32_t lane_base = taddr + (uint32_t(32 * (warp & 3)) << 16);
#pragma unroll
            for (int h4 = 0; h4 < 16; h4 += 4) {
                const int i = ib + h4;
                if (i >= ie) break;
                uint32_t s[16];
                asm volatile(
                    "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, "
                    "%13, %14, %15}, [%16];"
                    : "=r"(s[0]), "=r"(s[1]), "=r"(s[2]), "=r"(s[3]), "=r"(s[4]), "=r"(s[5]), "=r"(s[6]), "=r"(s[7]),
                      "=r"(s[8]), "=r"(s[9]), "=r"(s[10]), "=r"(s[11]), "=r"(s[12]), "=r"(s[13]), "=r"(s[14]),
                      "=r"(s[15])
                    : "r"(lane_base + uint32_t(4 * (i - ig))));
                // all four (primes up to k rounded up to four have weights, constants and rows)
                const uint4 c01 = *reinterpret_cast<const uint4*>(s_pc + i), c23 = *reinterpret_cast<const uint4*>(s_pc + i + 2);
                const uint32_t p[4] = {c01.x, c01.z, c23.x, c23.z}, c48[4] = {c01.y, c01.w, c23.y, c23.w};
                uint32_t* rows = res_row(sB, i);
                asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
                for (int e = 0; e < 4; ++e)
                    rows[128 * e + (CC ? slot[e] : res_slot(i0 + i + e, m, C))] = fold_planes(s + 4 * e, p[e], c48[e]);
            }
        }
        asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
        __syncthreads();  // this pass's reads are done before the next MMA
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    }
    if (warp == 0)
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(kDecTcCols) : "memory");
    if (!ok) {
        report_stuck(t);
        return;
    }
    dec32_columns<LOG_N1, CC, LN2>(R, t.fwd32, s_pc, sB, N, N2, logC, j0, i0, i1);
}

// The item by its tile width and row length.
template <int LOG_N1>
__device__ __forceinline__ void dec_tc32_any(const ProductDesc& d, const Tables& t, int operand, int tile, int i0, int i1,
                                             bool early, uint8_t* smem, uint64_t (&bar)[2], uint32_t& taddr_slot) {
    if (LOG_N1 <= 4 && d.logN == 12 + LOG_N1)
        dec_tc32_item<LOG_N1, (kDecTcRows >> LOG_N1), 12>(d, t, operand, tile, i0, i1, early, smem, bar, taddr_slot);
    else if (d.logN >= 7)
        dec_tc32_item<LOG_N1, (kDecTcRows >> LOG_N1), 0>(d, t, operand, tile, i0, i1, early, smem, bar, taddr_slot);
    else
        dec_tc32_item<LOG_N1, 0, 0>(d, t, operand, tile, i0, i1, early, smem, bar, taddr_slot);
}

// What bounds it: issue slots (the five-instruction fold of every residue, the column butterflies)
// and the latency of a tile's phases, which four CTAs an SM overlap in part; DRAM and the tensor cores
// are idle most of the time. Two operands of N = 65536, 868 bits: 34.8 -> 25.9 us (a fold of five
// instructions, neighbouring columns a thread, one polling warp, one bulk copy of
// the weights).
//
// Four CTAs per SM, as k_dec_tc (tensor memory holds four of 128 columns). With `split`, a CTA takes
// one pass of 32 primes of its tile instead of all of them (small grids: every pass is then a CTA
// of its own).
template <int LOG_N1>
__global__ void __launch_bounds__(kThreads, 4) k_dec_tc32(ProductDesc d, Tables t, int first_operand, int tile0,
                                                           int tiles, int split, int early) {
#if NC_HAS_TCGEN05
    extern __shared__ __align__(16) uint8_t smem[];
    __shared__ uint64_t bar[2];
    __shared__ uint32_t taddr_slot;
    int b = int(blockIdx.x), i0 = 0, i1 = int(d.k);
    if (split) {
        const int passes = (i1 + kDecTc32PassPrimes - 1) / kDecTc32PassPrimes;
        i0 = (b % passes) * kDecTc32PassPrimes;
        if (i1 > i0 + kDecTc32PassPrimes) i1 = i0 + kDecTc32PassPrimes;
        b /= passes;
    }
    dec_tc32_any<LOG_N1>(d, t, first_operand + b / tiles, tile0 + b % tiles, i0, i1, early != 0, smem, bar, taddr_slot);
#endif
}

// ------------------------------------------------------------------------------------------
// CRT: inverse column stages into A (the raw residues' 4 bytes at K offset 4 i), the contraction
// with the plan's table (crt32_table, hostmath.h) and the one-word quotient.
//
// With r_i in [0, 2p_i) the residue of the transform (still to be multiplied by y_i), byte a of
// r_i has the weight E_{i,a} = (2^(8a) y_i mod p_i) (M/p_i), so x = sum r_{i,a} E_{i,a} - K M with
// K = round(sum r_{i,a} phi_{i,a}), phi = (2^(8a) y_i mod p_i) / p_i: the table holds E mod q and
// phi, so neither the product r_i y_i nor a separate quotient sum is left to the integer pipes. The
// byte sums are below 4 * 64 * 255^2 < 2^24; K is exact because |x| < M / 8 and the floors of 256
// terms lose less than 255 * 256 / 2^32 (phi has 32 bits); and T = sum r_{i,a} (E mod q) +
// K ((-M) mod q) < 2^17 q, whose quotient by q is one word.
//
// What bounds it: the column butterflies and loads (59 residues of a coefficient against one
// contraction row), so integer issue and load latency, not the tensor cores. 128-coefficient tiles
// with the primes in passes of 32 through one 20 KB A buffer keep a CTA at 54 KB, four per SM.
// N = 65536, 868 bits: 24.6 -> 19.7 us a stage; N = 1024, where the old CRT was a chain of 59 dependent
// loads a thread in four CTAs: 32.8 -> 16.0 us a product.

// A: [16 row groups][8 K chunks of four primes][8 rows][16 B], the chunks 16 or 32 bytes and the row
// groups 16 bytes further apart than packed: a warp's four-byte stores (eight groups of neighbouring
// columns x four primes, or four x eight) then fall on 32 banks.
template <int LOG_N1>
struct Crt32Layout {
    static constexpr int kChunk = LOG_N1 == 4 ? 144 : 160;
    static constexpr int kGroup = 8 * kChunk + 16;
    __device__ static int at(int row, int il) {
        return (row >> 3) * kGroup + (il >> 2) * kChunk + (row & 7) * 16 + (il & 3) * 4;
    }
};
constexpr int kCrt32ABytes = 16 * (8 * 160 + 16);

// Primes [i0, i0 + np) of the tile's 2^logC columns: N1 residues at stride N2 (2^LN2, or N / N1 with
// LN2 0), the inverse stages of the merged tree, four bytes each into A. A thread takes VJ neighbouring
// columns of a prime (16- or 8-byte loads, one set of twiddles and addresses); one-residue loads were most
// of the stage's instructions at small N1, and their latency its time. Tiles of fewer columns go one by one.
template <int LOG_N1, int LN2, int VJ>
__device__ __forceinline__ void crt32_columns(const uint32_t* res, const uint2* tw0, int logN, int logC, int np,
                                              const uint32_t* s_p, uint8_t* sA) {
    using A = Crt32Layout<LOG_N1>;
    constexpr int N1 = 1 << LOG_N1;
    const int N = 1 << logN;
    const int N2 = LN2 ? 1 << LN2 : N >> LOG_N1;
    const int C = 1 << logC;
    const int tid = int(threadIdx.x);
    if constexpr (LOG_N1 == 5) {
        // 32-point columns on two adjacent lanes (as crt_columns_tc): lane h loads rows
        // [16h, 16h + 16), runs the inverse stages of its half-subtree, and the last stage's pairs
        // (u, u + 16) are split between the lanes after one exchange of eight values
        const int total = 2 * np * C;
        const int lane = tid & 31;
        for (int w0 = tid & ~31; w0 < total; w0 += kThreads) {
            const int w = w0 + lane;
            const bool active = w < total;
            const int item = active ? w >> 1 : 0, h = w & 1;
            const int i = item >> logC, j = item & (C - 1);
            const uint32_t* row = res + size_t(i) * N + j + size_t(16 * h) * N2;
            uint32_t v[1][16];
#pragma unroll
            for (int u = 0; u < 16; ++u) v[0][u] = active ? __ldcg(row + size_t(u) * N2) : 0u;
            const uint32_t p = s_p[i], p2 = 2 * p;
            const uint2* tw = tw0 + size_t(i) * kMaxN;
            w32::column_inverse_root<4, 1>(tw, 2 + h, p, v);
            const uint2 w1 = __ldg(tw + 1);
#pragma unroll
            for (int e = 0; e < 8; ++e) {
                const uint32_t got = __shfl_xor_sync(0xffffffffu, h ? v[0][e] : v[0][8 + e], 1);
                uint32_t lo = h ? got : v[0][e], hi = h ? v[0][8 + e] : got;  // rows 8h + e and 8h + e + 16
                w32::gs_bfly(lo, hi, w1.x, w1.y, p, p2);
                if (active) {
                    *reinterpret_cast<uint32_t*>(sA + A::at((8 * h + e) * C + j, i)) = lo;
                    *reinterpret_cast<uint32_t*>(sA + A::at((8 * h + e + 16) * C + j, i)) = hi;
                }
            }
        }
    } else {
        constexpr int LV = VJ == 4 ? 2 : VJ == 2 ? 1 : 0;
        // lanes: up to eight groups of columns (2^logL) of one prime, then primes, then further groups
        const int logG = logC - LV, logL = logG < 3 ? logG : 3;
        const int primes = (np + 3) & ~3;
        const int total = primes << logG;
#pragma unroll 1
        for (int w = tid; w < total; w += kThreads) {
            const int low = w & ((1 << logL) - 1), mid = w >> logL;
            // mid walks the primes four at a time within each further run of 2^logL groups
            const int run = (mid >> 2) & ((1 << (logG - logL)) - 1);
            const int il = ((mid >> (2 + logG - logL)) << 2) + (mid & 3);
            const int j = ((run << logL) + low) << LV;
            if (il >= np) continue;
            const uint32_t* row = res + size_t(il) * N + j;
            uint32_t v[VJ][N1];
#pragma unroll
            for (int u = 0; u < N1; ++u) {
                if constexpr (VJ == 4) {
                    const uint4 q = __ldcg(reinterpret_cast<const uint4*>(row + size_t(u) * N2));
                    v[0][u] = q.x;
                    v[1][u] = q.y;
                    v[2][u] = q.z;
                    v[3][u] = q.w;
                } else if constexpr (VJ == 2) {
                    const uint2 q = __ldcg(reinterpret_cast<const uint2*>(row + size_t(u) * N2));
                    v[0][u] = q.x;
                    v[1][u] = q.y;
                } else {
                    v[0][u] = __ldcg(row + size_t(u) * N2);
                }
            }
            if (LOG_N1 > 0) w32::column_inverse_root<LOG_N1, VJ>(tw0 + size_t(il) * kMaxN, 1, s_p[il], v);
            if (logC >= 3) {
                // rows u C + j are a constant distance apart, and VJ neighbours lie in one row group
                uint8_t* at = sA + A::at(j, il);
                const int step = (C >> 3) * A::kGroup;
#pragma unroll
                for (int u = 0; u < N1; ++u)
#pragma unroll
                    for (int e = 0; e < VJ; ++e) *reinterpret_cast<uint32_t*>(at + u * step + 16 * e) = v[e][u];
            } else {
#pragma unroll
                for (int u = 0; u < N1; ++u)
#pragma unroll
                    for (int e = 0; e < VJ; ++e) *reinterpret_cast<uint32_t*>(sA + A::at(u * C + j + e, il)) = v[e][u];
            }
        }
    }
}

__device__ __forceinline__ void tmem_ld4(uint32_t (&s)[4], uint32_t addr) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x4.b32 {%0, %1, %2, %3}, [%4];"
                 : "=r"(s[0]), "=r"(s[1]), "=r"(s[2]), "=r"(s[3])
                 : "r"(addr));
}
__device__ __forceinline__ void tmem_ld8(uint32_t (&s)[8], uint32_t addr) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                 : "=r"(s[0]), "=r"(s[1]), "=r"(s[2]), "=r"(s[3]), "=r"(s[4]), "=r"(s[5]), "=r"(s[6]), "=r"(s[7])
                 : "r"(addr));
}
__device__ __forceinline__ void tmem_wait_ld() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }

// Constants of the finish in shared memory, each padded to whole 16-byte words.
constexpr int kCrt32Words = 36;

// This thread's coefficient from its lane of the accumulator, T mod q, to L limbs at `o` (if `store`).
// All the lanes of a warp together (tensor-memory loads).
template <int LW>
__device__ __forceinline__ void crt32_finish(const QConst32* qc, const uint32_t* s_consts, uint32_t lane_base, int L,
                                             uint32_t* o, bool store) {
    const uint32_t *s_negm = s_consts, *s_nq = s_consts + kCrt32Words, *s_q = s_consts + 2 * kCrt32Words;
    uint32_t r[LW + 1];
    const int c0 = int(__ldg(&qc->top_byte)), sh = __ldg(&qc->top_shift);
    uint32_t ph[4], top[8];
    tmem_ld4(ph, lane_base + uint32_t(4 * LW));
    tmem_ld8(top, lane_base + uint32_t(c0));
    tmem_wait_ld();
    const uint64_t phi = mad_wide(ph[3], 1u << 24, mad_wide(ph[2], 1u << 16, mad_wide(ph[1], 1u << 8, uint64_t(ph[0]))));
    const uint32_t kq = uint32_t((phi + (1ull << 31)) >> 32);
    // bytes c0 .. c0 + 4 of T (the bytes below add less than 2^18 units of 2^(8 c0), against
    // q >= 2^(32 + 8 c0) where c0 > 0), then its 31 leading bits
    uint64_t vt = mad_wide(top[3], 1u << 24, mad_wide(top[2], 1u << 16, mad_wide(top[1], 1u << 8, uint64_t(top[0])))) +
                  (uint64_t(top[4]) << 32);
    vt += uint64_t(kq) * __ldg(&qc->top_neg_m);
    const uint32_t y = uint32_t(sh >= 0 ? vt >> sh : vt << -sh);
    const uint32_t qh = __umulhi(y, __ldg(&qc->mu1)) >> 13;  // floor(T / q) or one less
    // T - qh q = sum of bytes + kq ((-M) mod q) + qh (2^(32 (LW + 1)) - q), one carry pass; the next
    // columns are on their way while two words are formed
    uint64_t carry = 0;
    uint32_t s[2][8];
    tmem_ld8(s[0], lane_base);
    tmem_wait_ld();
#pragma unroll
    for (int g = 0; g < LW / 2; ++g) {
        if (g + 1 < LW / 2) tmem_ld8(s[(g + 1) & 1], lane_base + uint32_t(8 * (g + 1)));
        const uint32_t* sg = s[g & 1];
#pragma unroll
        for (int e = 0; e < 2; ++e) {
            const int w = 2 * g + e;
            const uint32_t lo = sg[4 * e] + (sg[4 * e + 1] << 8), hi = sg[4 * e + 2] + (sg[4 * e + 3] << 8);
            const uint64_t own = mad_wide(hi, 1u << 16, mad_wide(qh, s_nq[w], mad_wide(kq, s_negm[w], uint64_t(lo))));
            carry += own;
            r[w] = uint32_t(carry);
            carry >>= 32;
        }
        if (g + 1 < LW / 2) tmem_wait_ld();
    }
    r[LW] = uint32_t(mad_wide(qh, 0xffffffffu, carry));
    // r < 2q: the leading two words decide, except for about one coefficient in 2^12
    const uint64_t rt = (uint64_t(r[LW - 1]) << 32) | r[LW - 2], qt = (uint64_t(s_q[LW - 1]) << 32) | s_q[LW - 2];
    if (r[LW] != 0 || rt >= qt) {
        uint32_t b = 0;
#pragma unroll
        for (int w = 0; w < LW; ++w) {
            const uint64_t df = uint64_t(r[w]) - s_q[w] - b;
            b = uint32_t(df >> 32) & 1u;
        }
        if (r[LW] >= b) {
            b = 0;
#pragma unroll
            for (int w = 0; w < LW; ++w) {
                const uint64_t df = uint64_t(r[w]) - s_q[w] - b;
                r[w] = uint32_t(df);
                b = uint32_t(df >> 32) & 1u;
            }
        }
    }
    if (!store) {
        // rows beyond a tile of fewer than 32
    } else if ((L & 3) == 0) {
#pragma unroll
        for (int l = 0; l < LW; l += 4)
            if (l < L) *reinterpret_cast<uint4*>(o + l) = make_uint4(r[l], r[l + 1], r[l + 2], r[l + 3]);
    } else if ((L & 1) == 0) {
#pragma unroll
        for (int l = 0; l < LW; l += 2)
            if (l < L) *reinterpret_cast<uint2*>(o + l) = make_uint2(r[l], r[l + 1]);
    } else {
#pragma unroll
        for (int l = 0; l < LW; ++l)
            if (l < L) o[l] = r[l];
    }
}

// By LW, not inlined: one copy serves the kernels of every column length, and at the call next to
// nothing of theirs is live.
__device__ __noinline__ void crt32_finish_any(int LW, const QConst32* qc, const uint32_t* s_consts, uint32_t lane_base,
                                              int L, uint32_t* o, bool store) {
    switch (LW) {
#define NC_CRT32_FINISH(n) \
    case n: crt32_finish<n>(qc, s_consts, lane_base, L, o, store); break;
        NC_LW_CASES(NC_CRT32_FINISH)
#undef NC_CRT32_FINISH
        default: break;
    }
}

// Shared memory: A (128 rows x the 128 K bytes of 32 primes; the output tile once the sums are
// out), the finish's constants, p of up to 64 primes, the plan's table; raised so that no more CTAs
// share an SM than its tensor memory holds.
NC_HD constexpr size_t crt_tc32_smem_bytes(int LW) {
    return smax(size_t(kCrt32ABytes) + crt32_table_bytes(LW) + size_t(kMaxPrimes32) * 4 + size_t(kCrt32Words) * 4 * 3,
                (size_t(233472) / (512 / crt32_tmem_cols(LW) + 1) + 16) / 16 * 16);
}

// The output tile (N1 segments of C consecutive coefficients) to its place in c: a warp a segment
// where there are as many segments as warps, else store_tile.
__device__ __forceinline__ void crt32_store(uint32_t* c, int N2, int L, int j0, int C, int N1, const uint32_t* s_out) {
    const int seg = C * L;
    if (N1 < kThreads / 32 || ((size_t(N2) * L | size_t(j0) * L | size_t(seg)) & 3) != 0) {
        store_tile(c, N2, L, j0, C, N1, s_out);
        return;
    }
    const int warp = int(threadIdx.x) >> 5, lane = int(threadIdx.x) & 31;
    for (int u = warp; u < N1; u += kThreads / 32) {
        uint4* dst = reinterpret_cast<uint4*>(c + (size_t(u) * N2 + j0) * L);
        const uint4* src = reinterpret_cast<const uint4*>(s_out + u * seg);
        for (int x = lane; x < (seg >> 2); x += 32) dst[x] = src[x];
    }
}

// One tile with every thread of a 256-thread CTA, columns of 2^LOG_N1 points at stride 2^LN2 (N / N1
// with LN2 0). The caller owns tensor-memory columns for the product's LW at `taddr` and
// two initialised mbarriers `bars` (the MMAs', the table's). False if one of them did not complete in time.
template <int LOG_N1, int LN2>
__device__ __forceinline__ bool crt32_coeffs_tc(const ProductDesc& d, const Tables& t, int tile, int logT,
                                                bool early, uint8_t* smem, uint32_t taddr, uint64_t* bars) {
    uint64_t* bar = bars;
    using A = Crt32Layout<LOG_N1>;
    // the descriptor's fields once (a batch's lies in global memory)
    const int LW = int(d.LW), NC = crt32_cols(LW), logN = int(d.logN);
    const uint32_t* ra = reinterpret_cast<const uint32_t*>(d.ra);
    uint32_t* const c_out = d.c;
    const int N = 1 << logN;
    const int N2 = LN2 ? 1 << LN2 : N >> LOG_N1;
    const int T = 1 << logT;
    const int logC = logT - LOG_N1, C = 1 << logC;
    const int k = int(d.k), L = int(d.L);
    const int j0 = tile * C;

    uint8_t* sA = smem;
    uint32_t* s_negm = reinterpret_cast<uint32_t*>(sA + kCrt32ABytes);
    uint32_t* s_nq = s_negm + kCrt32Words;
    uint32_t* s_q = s_nq + kCrt32Words;
    uint32_t* s_p = s_q + kCrt32Words;
    uint8_t* sB = reinterpret_cast<uint8_t*>(s_p + kMaxPrimes32);
    const int tid = int(threadIdx.x), warp = tid >> 5;

    const QConst32* qc = d.qc32;
    for (int w = tid; w < k; w += kThreads) s_p[w] = __ldg(&t.pc32[w].p);
    for (int w = tid; w < kMqStride; w += kThreads) {
        s_negm[w] = __ldg(qc->neg_m + w);
        s_nq[w] = __ldg(qc->neg_q + w);
        s_q[w] = __ldg(qc->q + w);
    }
    // the table is first read by the MMAs: its copy runs behind the column stages, and the thread that
    // issues them waits for it (its K bytes from 4 k up are zero, so A's are never read into the sums)
    if (tid == 0) bulk_table(sB, d.crt_b, uint32_t(NC) * 256u, smem_u32(bars + 1));
    __syncthreads();
    if (early) pdl_trigger();
    pdl_wait();  // the residues come from the stream's previous kernel
    pdl_trigger();

    const uint32_t bar_addr = smem_u32(bar);
    const int passes = (k + 31) >> 5;
#pragma unroll 1
    for (int g = 0; g < passes; ++g) {
        // the A buffer is free once the pass before has been read
        if (g > 0 &&
            !__syncthreads_and(warp != 0 || bar_wait(t, bar_addr, uint32_t((g - 1) & 1), kGiveUpMmas) ? 1 : 0))
            return false;
        const int i0 = 32 * g, np = k - i0 < 32 ? k - i0 : 32;
        const uint32_t* res = ra + size_t(i0) * N + j0;
        constexpr int VJ = column_width(LOG_N1);
        if (LOG_N1 == 5 || logC >= 3)
            crt32_columns<LOG_N1, LN2, VJ>(res, t.inv32 + size_t(i0) * kMaxN, logN, logC, np, s_p + i0, sA);
        else
            crt32_columns<LOG_N1, LN2, 1>(res, t.inv32 + size_t(i0) * kMaxN, logN, logC, np, s_p + i0, sA);
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
        if (!__syncthreads_and(tid != 0 || g > 0 || bar_wait(t, smem_u32(bars + 1), 0, kGiveUpCopies) ? 1 : 0)) return false;
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        if (tid == 0) {
            const uint32_t idesc = (2u << 4) | (uint32_t(NC >> 3) << 17) | (uint32_t(kCrt32Rows >> 4) << 24);
            const uint32_t a0 = smem_u32(sA), b0 = smem_u32(sB) + uint32_t(g) * 1024u;
            for (int s = 0; s < (4 * np + 31) / 32; ++s) {
                const uint64_t da = kmajor_desc(a0 + uint32_t(s) * 2u * A::kChunk, A::kChunk, A::kGroup);
                const uint64_t db = kmajor_desc(b0 + uint32_t(s) * 256u, 128u, 2048u);
                asm volatile(
                    "{\n\t.reg .pred p;\n\t"
                    "setp.ne.b32 p, %4, 0;\n\t"
                    "tcgen05.mma.cta_group::1.kind::i8 [%0], %1, %2, %3, p;\n\t}" ::"r"(taddr),
                    "l"(da), "l"(db), "r"(idesc), "r"(g + s));
            }
            asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar_addr)
                         : "memory");
        }
    }
    if (!__syncthreads_and(warp != 0 || bar_wait(t, bar_addr, uint32_t((passes - 1) & 1), kGiveUpMmas) ? 1 : 0)) return false;
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");

    // every MMA has read A: it takes the output tile
    uint32_t* s_out = reinterpret_cast<uint32_t*>(sA);
    if (32 * warp < T)
        crt32_finish_any(LW, qc, s_negm, taddr + (uint32_t(32 * warp) << 16), L, s_out + tid * L, tid < T);
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    crt32_store(c_out, N2, L, j0, C, 1 << LOG_N1, s_out);
    return true;
}

// The tile within a kernel: tensor memory (`cols` columns) and the mbarrier around it.
template <int LOG_N1>
__device__ __forceinline__ void crt32_cta(const ProductDesc& d, const Tables& t, int tile, int logT, uint32_t cols,
                                          bool early) {
    extern __shared__ __align__(16) uint8_t smem[];
    __shared__ uint64_t bars[2];  // the MMAs', the table's
    __shared__ uint32_t taddr_slot;
    if (threadIdx.x < 32) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&taddr_slot)),
                     "r"(cols)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    if (threadIdx.x == 0) {
        for (int e = 0; e < 2; ++e)
            asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_u32(bars + e)) : "memory");
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t taddr = taddr_slot;
    const bool ok = LOG_N1 <= 4 && d.logN == 12 + LOG_N1
                        ? crt32_coeffs_tc<LOG_N1, 12>(d, t, tile, logT, early, smem, taddr, bars)
                        : crt32_coeffs_tc<LOG_N1, 0>(d, t, tile, logT, early, smem, taddr, bars);
    if (!ok) report_stuck(t);
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (threadIdx.x < 32)
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(cols) : "memory");
}

template <int LOG_N1>
__global__ void __launch_bounds__(kThreads, 4) k_crt_tc32(ProductDesc d, Tables t, int logT, uint32_t cols,
                                                           int early) {
#if NC_HAS_TCGEN05
    crt32_cta<LOG_N1>(d, t, int(blockIdx.x), logT, cols, early != 0);
#endif
}

// ------------------------------------------------------------------------------------------
// row blocks

// What bounds it: the 32-bit multiply pipe in bursts (about 60% of cycles), and between them the waits
// for the staged twiddles and residues and for the other warps of a block. N = 65536, 868 bits,
// blocks of 4096: 47.3 -> 44.8 us (padded places, block barriers, additions off the multiply pipe).
// Resident CTAs per SM: radix-8 passes in 256-thread CTAs at four (64 registers: three and five CTAs
// are no faster at N = 2^16); radix 16 at two, which is what its shared memory (100 KB) lets in (its
// launch bound of three holds it to 80 registers).
template <int LOG_N2, int LOG_E, int THREADS>
__global__ void __launch_bounds__(THREADS, (THREADS == 256 ? (LOG_E == 3 ? 4 : 3) : 2)) k_row32(ProductDesc d, Tables t,
                                                                                                   int early) {
    extern __shared__ __align__(16) uint8_t smem[];
    __shared__ uint64_t bar;
    if (early) pdl_trigger();
    const uint32_t b = smem_u32(&bar);
    w32::row_barrier_init<LOG_N2, LOG_E, THREADS>(b);
    if (!w32::row_blocks<LOG_N2, LOG_E, THREADS>(d, t, int(blockIdx.x), smem, b, 0, true)) report_stuck(t);
}

#define NC_ROW32_VARIANTS(X)                                                                                   \
    X(1, 4, 256) X(2, 4, 256) X(3, 4, 256) X(4, 4, 256) X(5, 4, 256) X(6, 4, 256) X(7, 4, 256) X(8, 4, 256)  \
    X(9, 4, 256) X(10, 4, 256) X(11, 4, 256) X(12, 4, 256) X(6, 3, 256) X(7, 3, 256) X(8, 3, 256)           \
    X(9, 3, 256) X(10, 3, 256) X(11, 3, 256) X(12, 3, 512)

// ------------------------------------------------------------------------------------------
// batches (products of N < 2^15 on the 30-bit engine; batch.cu): the residue items of every such
// product (one CTA per item), then one persistent row launch per row-block size, then the CRT
// items. The launches of a batch run in stream order, so no item waits on another.

// Residue items (x = product, y = operand * tiles_tc + tile), every product of the launch with
// column length 2^LOG_N1.
template <int LOG_N1>
__global__ void __launch_bounds__(kThreads, 4) k_batch_dec_tc32(BatchCrtArgs a) {
#if NC_HAS_TCGEN05
    extern __shared__ __align__(16) uint8_t smem[];
    __shared__ uint64_t bar[2];
    __shared__ uint32_t taddr_slot;
    const uint2 w = __ldg(a.items + blockIdx.x);
    const BatchProduct& bp = a.products[w.x];
    const int tiles = int(bp.tiles_tc);
    const int operand = int(bp.first_operand) + int(w.y) / tiles, tile = int(w.y) % tiles;
    dec_tc32_any<LOG_N1>(bp.d, a.tables, operand, tile, 0, int(bp.d.k), false, smem, bar, taddr_slot);
#endif
}

// Row items (x = product, y = row-CTA index) with row blocks of 2^LOG_N2, radix 8, 256 threads:
// persistent CTAs take items in queue order; each item's twiddles and residue blocks arrive on the
// CTA's mbarrier, one phase per item. Bound as k_row32 is, without its last wave (64 x 16384, 868 bits:
// 481 -> 437 us with padded places, block barriers and additions off the multiply pipe).
template <int LOG_N2>
__global__ void __launch_bounds__(kThreads, 4) k_persistent_rows32(BatchArgs a) {
    extern __shared__ __align__(16) uint8_t smem[];
    __shared__ uint64_t bar;
    __shared__ int s_item;
    __shared__ __align__(16) BatchProduct s_bp;
    constexpr int kWords = int(sizeof(BatchProduct) / 4);
    // with one row block a CTA, items come two at a time: a mirror pair (adjacent in the queue,
    // batch.cu) runs as row_pair, anything else as two row_blocks
    constexpr bool kPairs = RowShape<LOG_N2, kBatchRowLogE>::T == kThreads;
    pdl_trigger();
    const uint32_t b = smem_u32(&bar);
    row_barrier_init<LOG_N2, kBatchRowLogE, kThreads>(b);
    uint32_t parity = 0;
    bool ok = true;
    auto load_product = [&](uint32_t x) {
        if (threadIdx.x < kWords)
            reinterpret_cast<uint32_t*>(&s_bp)[threadIdx.x] =
                __ldg(reinterpret_cast<const uint32_t*>(a.products + (x & 0x0fffffffu)) + threadIdx.x);
        __syncthreads();
    };
    auto single = [&](int y) {
        ok = row_blocks<LOG_N2, kBatchRowLogE, kThreads>(s_bp.d, a.tables, y, smem, b, parity);
        parity ^= 1u;
    };
    for (;;) {
        if (threadIdx.x == 0) s_item = int(atomicAdd(a.head, kPairs ? 2u : 1u));
        __syncthreads();
        const int it = s_item;
        if (it >= a.n_items) break;
        const uint2 w = __ldg(a.items + it);
        load_product(w.x);
        if constexpr (kPairs) {
            const bool has2 = it + 1 < a.n_items;
            const uint2 w2 = has2 ? __ldg(a.items + it + 1) : make_uint2(0u, 0u);
            const int logN1 = int(s_bp.d.logN) - LOG_N2;
            const int mask = (1 << logN1) - 1;
            const int mirror = (int(w.y) & ~mask) | (mask - (int(w.y) & mask));
            if (has2 && w2.x == w.x && s_bp.d.mode == kModeProduct && logN1 >= 1 && int(w2.y) == mirror) {
                // two phases, so the parity is unchanged
                ok = row_pair<LOG_N2, kBatchRowLogE, kThreads>(s_bp.d, a.tables, int(w.y), int(w2.y), smem, b, parity);
            } else {
                single(int(w.y));
                if (ok && has2) {
                    __syncthreads();  // s_bp is rewritten
                    load_product(w2.x);
                    single(int(w2.y));
                }
            }
        } else {
            single(int(w.y));
        }
        if (!ok) {
            report_stuck(a.tables);
            break;
        }
        __syncthreads();  // s_item and s_bp are rewritten by the next round
    }
}

// CRT items (x = product, y = tile) of the products with column length 2^LOG_N1.
template <int LOG_N1>
__global__ void __launch_bounds__(kThreads, 4) k_batch_crt_tc32(BatchCrtArgs a, uint32_t cols) {
#if NC_HAS_TCGEN05
    const uint2 w = __ldg(a.items + blockIdx.x);
    const ProductDesc& d = a.products[w.x].d;
    crt32_cta<LOG_N1>(d, a.tables, int(w.y), crt32_batch_log_tile(int(d.logN)), cols, false);
#endif
}

void* batch_dec_tc32_kernel(int logN1) {
    switch (logN1) {
        case 0: return reinterpret_cast<void*>(&k_batch_dec_tc32<0>);
        case 1: return reinterpret_cast<void*>(&k_batch_dec_tc32<1>);
        case 2: return reinterpret_cast<void*>(&k_batch_dec_tc32<2>);
        case 3: return reinterpret_cast<void*>(&k_batch_dec_tc32<3>);
        case 4: return reinterpret_cast<void*>(&k_batch_dec_tc32<4>);
        case 5: return reinterpret_cast<void*>(&k_batch_dec_tc32<5>);
        default: return nullptr;
    }
}

void* persistent_rows32_kernel(int logN2) {
    switch (logN2) {
#define NC_P_ROWS32(n) \
    case n: return reinterpret_cast<void*>(&k_persistent_rows32<n>);
        NC_P_ROWS32(1) NC_P_ROWS32(2) NC_P_ROWS32(3) NC_P_ROWS32(4) NC_P_ROWS32(5) NC_P_ROWS32(6)
        NC_P_ROWS32(7) NC_P_ROWS32(8) NC_P_ROWS32(9) NC_P_ROWS32(10) NC_P_ROWS32(11)
#undef NC_P_ROWS32
        default: return nullptr;
    }
}

void* dec_tc32_kernel(int logN1) {
    switch (logN1) {
        case 0: return reinterpret_cast<void*>(&k_dec_tc32<0>);
        case 1: return reinterpret_cast<void*>(&k_dec_tc32<1>);
        case 2: return reinterpret_cast<void*>(&k_dec_tc32<2>);
        case 3: return reinterpret_cast<void*>(&k_dec_tc32<3>);
        case 4: return reinterpret_cast<void*>(&k_dec_tc32<4>);
        case 5: return reinterpret_cast<void*>(&k_dec_tc32<5>);
        default: return nullptr;
    }
}

void* crt_tc32_kernel(int logN1) {
    switch (logN1) {
        case 0: return reinterpret_cast<void*>(&k_crt_tc32<0>);
        case 1: return reinterpret_cast<void*>(&k_crt_tc32<1>);
        case 2: return reinterpret_cast<void*>(&k_crt_tc32<2>);
        case 3: return reinterpret_cast<void*>(&k_crt_tc32<3>);
        case 4: return reinterpret_cast<void*>(&k_crt_tc32<4>);
        case 5: return reinterpret_cast<void*>(&k_crt_tc32<5>);
        default: return nullptr;
    }
}

void* batch_crt_tc32_kernel(int logN1) {
    switch (logN1) {
        case 0: return reinterpret_cast<void*>(&k_batch_crt_tc32<0>);
        case 1: return reinterpret_cast<void*>(&k_batch_crt_tc32<1>);
        case 2: return reinterpret_cast<void*>(&k_batch_crt_tc32<2>);
        case 3: return reinterpret_cast<void*>(&k_batch_crt_tc32<3>);
        case 4: return reinterpret_cast<void*>(&k_batch_crt_tc32<4>);
        case 5: return reinterpret_cast<void*>(&k_batch_crt_tc32<5>);
        default: return nullptr;
    }
}

}  // namespace

}  // namespace w32

// Which kernels of a plain product release the next one before their own wait (after it otherwise).
// Early, the launch latencies of short kernels overlap; but the kernels of two products are then resident
// at once and their CTAs placed unevenly, which costs more once kernels are longer. Early where that
// measured faster (us a product, after the wait and early):
// - up to N = 32, where a kernel has one CTA or few: N = 16, 31 bits 16.5 and 12.7, 868 bits 19.5 and
//   17.1; N = 64, 434 bits 11.2 and 11.1, 600 bits at N = 128 11.3 and 11.7;
// - rows and CRT from N = 2^14 up to 16 primes: at 2^14, 31 bits 18.1 and 15.0, 130 bits 19.2 and 17.1;
//   at 2^16, 31 bits 21.8 and 20.7; but 200 bits at 2^13 12.9 and 14.0, 300 bits (21 primes) at 2^15
//   21.9 and 22.5.
enum : int { kEarlyDec = 1, kEarlyRow = 2, kEarlyCrt = 4 };
static int early_triggers(int logN, int k) {
    if (logN <= 5) return kEarlyDec | kEarlyRow | kEarlyCrt;
    return logN >= 14 && k <= 16 ? kEarlyRow | kEarlyCrt : 0;
}

// Residue launches of at most this many CTAs give each pass of primes its own CTA.
constexpr int kDec32SplitCtas = 74;

// Shared memory of the 30-bit residue stage: the limb tile, the weights of the primes it
// copies and their constants; raised, as dec_tc_smem_bytes, to keep four CTAs per SM.
size_t dec_tc32_smem_bytes(int k) {
    return smax(size_t(kDecTcRows) * 128 + size_t(w32::dec32_weight_pairs(k)) * 1024 + size_t(kMaxPrimes32) * 16,
                (size_t(233472) / (512 / kDecTcCols + 1) + 16) / 16 * 16);
}

void* row32_kernel(const RowConfig& c) {
#define NC_ROW32(n, e, th) \
    if (c.logN2 == n && c.logE == e && c.threads == th) return reinterpret_cast<void*>(&w32::k_row32<n, e, th>);
    NC_ROW32_VARIANTS(NC_ROW32)
#undef NC_ROW32
    return nullptr;
}

std::vector<RowConfig> all_row32_variants() {
    std::vector<RowConfig> v;
#define NC_ROW32_LIST(n, e, th) v.push_back(RowConfig{n, e, th});
    NC_ROW32_VARIANTS(NC_ROW32_LIST)
#undef NC_ROW32_LIST
    return v;
}

cudaError_t prepare_w32() {
    cudaError_t e = cudaSuccess;
    for (const RowConfig& c : all_row32_variants()) {
        if (e != cudaSuccess) break;
        e = cudaFuncSetAttribute(row32_kernel(c), cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 int(w32::row_smem_bytes(c.threads, c.logE)));
    }
    for (int l = 0; l <= kMaxLogN1 && e == cudaSuccess; ++l)
        e = cudaFuncSetAttribute(w32::dec_tc32_kernel(l), cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 int(dec_tc32_smem_bytes(kMaxPrimes32)));
    for (int l = 0; l <= kMaxLogN1 && e == cudaSuccess; ++l)
        e = cudaFuncSetAttribute(w32::crt_tc32_kernel(l), cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 int(w32::crt_tc32_smem_bytes(kMaxL)));
    for (int l = 0; l <= kMaxLogN1 && e == cudaSuccess; ++l)
        e = cudaFuncSetAttribute(w32::batch_dec_tc32_kernel(l), cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 int(dec_tc32_smem_bytes(kMaxPrimes32)));
    for (int n = 1; n <= kBatchRowLogMax && e == cudaSuccess; ++n)
        e = cudaFuncSetAttribute(w32::persistent_rows32_kernel(n), cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 int(w32::row_smem_bytes(kThreads, kBatchRowLogE)));
    for (int l = 0; l <= kMaxLogN1 && e == cudaSuccess; ++l)
        e = cudaFuncSetAttribute(w32::batch_crt_tc32_kernel(l), cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 int(w32::crt_tc32_smem_bytes(kMaxL)));
    return e;
}

cudaError_t launch_batch_dec_tc32(const BatchCrtArgs& args, int logN1, int kmax, cudaStream_t s) {
    void* fn = w32::batch_dec_tc32_kernel(logN1);
    if (!fn) return cudaErrorInvalidValue;
    BatchCrtArgs a = args;
    void* params[] = {&a};
    return launch_pdl(fn, args.n_items, kThreads, dec_tc32_smem_bytes(kmax), s, params);
}

cudaError_t launch_persistent_rows32(const BatchArgs& args, int logN2, int ctas, cudaStream_t s) {
    void* fn = w32::persistent_rows32_kernel(logN2);
    if (!fn) return cudaErrorInvalidValue;
    BatchArgs a = args;
    void* params[] = {&a};
    return launch_pdl(fn, ctas, kThreads, w32::row_smem_bytes(kThreads, kBatchRowLogE), s, params);
}

cudaError_t persistent_rows32_occupancy(int logN2, int* ctas_per_sm) {
    void* fn = w32::persistent_rows32_kernel(logN2);
    if (!fn) return cudaErrorInvalidValue;
    return cudaOccupancyMaxActiveBlocksPerMultiprocessor(ctas_per_sm, fn, kThreads,
                                                         w32::row_smem_bytes(kThreads, kBatchRowLogE));
}

cudaError_t launch_batch_crt_tc32(const BatchCrtArgs& args, int logN1, int lw_max, cudaStream_t s) {
    void* fn = w32::batch_crt_tc32_kernel(logN1);
    if (!fn) return cudaErrorInvalidValue;
    BatchCrtArgs a = args;
    uint32_t cols = crt32_tmem_cols(lw_max);
    void* params[] = {&a, &cols};
    return launch_pdl(fn, args.n_items, kThreads, w32::crt_tc32_smem_bytes(lw_max), s, params);
}

cudaError_t launch_residues32(const ProductDesc& d, const Tables& t, int logN1, cudaStream_t s, int first, int count,
                              int tile0, int tiles) {
    void* fn = w32::dec_tc32_kernel(logN1);
    if (!fn || !t.res_w32 || int(d.k) > kMaxPrimes32) return cudaErrorInvalidValue;
    ProductDesc dd = d;
    Tables tt = t;
    // a pass of 32 primes a CTA while that leaves half the SMs free: the passes of a tile then run
    // side by side (868 bits, N = 1024: 16.4 -> 15.3 us a product; N = 4096, 128 CTAs and a short
    // second pass at 600 bits: 18.2 -> 22.6 us, so not there)
    const int passes = (int(d.k) + kDecTc32PassPrimes - 1) / kDecTc32PassPrimes;
    int split = count * tiles * passes <= kDec32SplitCtas ? 1 : 0;
    const int primes = split && int(d.k) > kDecTc32PassPrimes ? kDecTc32PassPrimes : int(d.k);
    int early = early_triggers(int(d.logN), int(d.k)) & kEarlyDec;
    void* args[] = {&dd, &tt, &first, &tile0, &tiles, &split, &early};
    return launch_pdl(fn, count * tiles * (split ? passes : 1), kThreads, dec_tc32_smem_bytes(primes), s, args);
}

cudaError_t launch_row32(const ProductDesc& d, const Tables& t, const RowConfig& cfg, cudaStream_t s) {
    void* fn = row32_kernel(cfg);
    if (!fn) return cudaErrorInvalidValue;
    const Geometry g = geometry(int(d.logN), int(d.k), cfg);
    ProductDesc dd = d;
    Tables tt = t;
    int early = early_triggers(int(d.logN), int(d.k)) & kEarlyRow;
    void* args[] = {&dd, &tt, &early};
    return launch_pdl(fn, g.row_ctas, cfg.threads, w32::row_smem_bytes(cfg.threads, cfg.logE), s, args);
}

cudaError_t launch_crt32(const ProductDesc& d, const Tables& t, cudaStream_t s) {
    const int logN1 = int(d.logN) - int(d.logN2);
    void* fn = w32::crt_tc32_kernel(logN1);
    if (!fn || !d.crt_b || !d.qc32) return cudaErrorInvalidValue;
    ProductDesc dd = d;
    Tables tt = t;
    int logT = crt32_log_tile(int(d.logN), logN1);
    uint32_t cols = crt32_tmem_cols(int(d.LW));
    int early = early_triggers(int(d.logN), int(d.k)) & kEarlyCrt;
    void* args[] = {&dd, &tt, &logT, &cols, &early};
    return launch_pdl(fn, 1 << (int(d.logN) - logT), kThreads, w32::crt_tc32_smem_bytes(int(d.LW)), s, args);
}

}  // namespace nc
