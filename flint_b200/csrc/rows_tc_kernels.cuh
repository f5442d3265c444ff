// Row pass with its length-32 transforms on the tensor cores.
//
// The row kernel's forward transforms end, and its inverse transform begins,
// with five levels on 32 consecutive positions and no twiddle after (before)
// them: a product with one fixed 32 x 32 matrix (tcgen05.cuh).  Here those
// levels are byte-matrix products: the strided levels leave an item of 2^13
// words as 256 rows of 32 residues, two 128-row A tiles, and the sums come back
// from TMEM to the thread that owns the row.
//
// What bounds it: issue slots and latency at 16 warps per SM (2^13-point rows of a
// 2^23-point product: issue 53% of cycles, FMA-heavy pipe 53%, ALU 48%, tensor pipe
// 8%; 159 instructions a point against 168): the five levels cost 9 instructions a
// word for tc_reduce instead of 15 of butterflies.  512 threads of 16 words at 64
// registers were slower (834 against 705 us on a 2^24-point product: the second
// vector of a strided pass no longer fits, so its twiddles are loaded twice).
//
// Row buffers hold position pos at word tc_swz(pos), which is the operand
// layout and needs no padding: every strided access of a warp is 32 consecutive
// positions, one swizzled 128-byte row, and 16-byte copies land in place.
#pragma once
#include "mpn_kernels.cuh"

namespace fb {

constexpr int TC_WORDS = 1 << 13;              // words per item (nv rows of C)
constexpr int TC_THREADS = TC_WORDS / 32;
constexpr int TC_COLS = 256;                   // TMEM columns: two tiles of 128
// b, two a buffers, W, barrier and TMEM address
constexpr size_t TC_ROWS_SMEM = (size_t)3 * TC_WORDS * 4 + TC_W_BYTES + 64;

// word offset of element m of a strided sub-transform from its element 0 at
// position `base` (row rb = base >> 5): a constant where the rows are 8 or
// more apart, else (32 apart, rb a multiple of 8) the chunk exchange of row m
template <int S>
__device__ __forceinline__ int tc_off(int base, int m)
{
    static_assert(S >= 256 || S == 32, "unsupported pass stride");
    if constexpr (S >= 256) return tc_swz(base) + m * S;
    else return (base ^ ((m & 7) << 2)) + m * 32;
}

// The levels of gs_strided_level2 / gs_strided; the last one (half-size 32) feeds
// the byte-matrix product, which takes any 32-bit representative: sums below 2 p
// and unreduced Shoup products, two instructions a butterfly less.
template <int Q, int H, int t, int NVEC>
__device__ __forceinline__ void tc_gs_level(uint32_t (&x)[1 << Q], uint32_t (&y)[NVEC == 2 ? 1 << Q : 1],
                                            const uint2* __restrict__ tw, int jj0, uint32_t p)
{
    constexpr int E = 1 << Q;
    constexpr int S = H >> (Q - 1);
    constexpr int hm = E >> (t + 1);
    constexpr int ht = H >> t;
    uint2 w[hm];
#pragma unroll
    for (int k = 0; k < hm; k++) w[k] = tw[ht + jj0 + k * S];
    auto bfly = [&](uint32_t& a, uint32_t& b, const uint2& v) {
        if constexpr (ht > 32) {
            bfly_gs<ROW_GS_FMA_ADDS>(a, b, v.x, v.y, p);
        } else {
            const uint32_t d = a - b + p;
            a = a + b;
            b = mul_shoup_lazy(d, v.x, v.y, p);
        }
    };
#pragma unroll
    for (int m = 0; m < E; m++)
        if ((m & hm) == 0) {
            bfly(x[m], x[m + hm], w[m & (hm - 1)]);
            if constexpr (NVEC == 2) bfly(y[m], y[m + hm], w[m & (hm - 1)]);
        }
    if constexpr (t + 1 < Q) tc_gs_level<Q, H, t + 1, NVEC>(x, y, tw, jj0, p);
}

// strided Gentleman-Sande passes of nv rows of 2^LOGL words, as gs_passes
template <int LOGL, int NVEC, int QMAX, int H, int REM>
__device__ __forceinline__ void tc_gs_passes(uint32_t* sx, uint32_t* sy, int nv, const uint2* __restrict__ tw,
                                             uint32_t p)
{
    if constexpr (REM > 0) {
        constexpr int Q = balanced_pass<REM, QMAX>();
        constexpr int E = 1 << Q, S = H >> (Q - 1), NSUB = (1 << LOGL) / E;
#pragma unroll 1
        for (int f = threadIdx.x; f < nv * NSUB; f += TC_THREADS) {
            const int s = f & (NSUB - 1), v = f / NSUB;
            const int jj0 = s & (S - 1);
            const int base = (v << LOGL) + (s / S) * (2 * H) + jj0;
            uint32_t x[E], y[NVEC == 2 ? E : 1];
#pragma unroll
            for (int m = 0; m < E; m++) {
                x[m] = sx[tc_off<S>(base, m)];
                if constexpr (NVEC == 2) y[m] = sy[tc_off<S>(base, m)];
            }
            tc_gs_level<Q, H, 0, NVEC>(x, y, tw, jj0, p);
#pragma unroll
            for (int m = 0; m < E; m++) {
                sx[tc_off<S>(base, m)] = x[m];
                if constexpr (NVEC == 2) sy[tc_off<S>(base, m)] = y[m];
            }
        }
        if constexpr (REM > Q) {
            __syncthreads();
            tc_gs_passes<LOGL, NVEC, QMAX, (H >> Q), REM - Q>(sx, sy, nv, tw, p);
        }
    }
}

// strided Cooley-Tukey passes; the last one stores to out (rows u < nrows only)
template <int LOGL, int QMAX, int H, int REM>
__device__ __forceinline__ void tc_ct_passes_out(uint32_t* sm, int nv, int nrows, const uint2* __restrict__ twi,
                                                 uint32_t p, uint32_t* __restrict__ out)
{
    constexpr int Q = balanced_pass<REM, QMAX>();
    constexpr int E = 1 << Q, S = H, NSUB = (1 << LOGL) / E;
#pragma unroll 1
    for (int f = threadIdx.x; f < nv * NSUB; f += TC_THREADS) {
        const int s = f & (NSUB - 1), v = f / NSUB;
        const int jj0 = s & (S - 1);
        const int base = (v << LOGL) + (s / S) * (S * E) + jj0;
        uint32_t x[E];
#pragma unroll
        for (int m = 0; m < E; m++) x[m] = sm[tc_off<S>(base, m)];
        ct_strided<Q, H, ROW_CT_FMA_ADDS>(x, twi, jj0, p);
        if constexpr (REM > Q) {
#pragma unroll
            for (int m = 0; m < E; m++) sm[tc_off<S>(base, m)] = x[m];
        } else if (v < nrows) {
#pragma unroll
            for (int m = 0; m < E; m++) out[base + m * S] = x[m];
        }
    }
    if constexpr (REM > Q) {
        __syncthreads();
        tc_ct_passes_out<LOGL, QMAX, (H << Q), REM - Q>(sm, nv, nrows, twi, p, out);
    }
}

// rows u0 .. u0 + nv - 1 (contiguous; zeros from row R on) into a row buffer
template <int LOGC>
__device__ __forceinline__ void tc_prefetch(uint32_t* dst, const uint32_t* __restrict__ base, int u0, int nv, int R)
{
    const uint32_t* src = base + ((size_t)u0 << LOGC);
    const int words = min(nv, R - u0) << LOGC;
#pragma unroll
    for (int k = 0; k < TC_WORDS / 4 / TC_THREADS; k++) {
        const int pos = 4 * (threadIdx.x + k * TC_THREADS);
        const unsigned d = tc_smem(dst + tc_swz(pos));
        const int n = pos < words ? 16 : 0;   // a zero source size fills with zeros
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(d), "l"(src + (n ? pos : 0)), "r"(n));
    }
    cp_async_commit();
}

// As k_rows (same arguments and results), for items of nv 2^LOGC = 2^13 words;
// grid = min(items, resident CTAs), block = 256, smem = TC_ROWS_SMEM.
template <int LOGC>
__global__ void __launch_bounds__(TC_THREADS, 2)
k_rows_tc(DevTables T, uint32_t* __restrict__ ra, const uint32_t* __restrict__ rb, int logR, int nv, int np,
          const uint32_t* __restrict__ scale, int squaring, const InstDesc* __restrict__ desc, int ninst, int rows)
{
    extern __shared__ __align__(1024) uint32_t sm[];
    uint32_t* const sb = sm;
    uint32_t* const sw = sm + 3 * TC_WORDS;
    uint64_t* const bar = reinterpret_cast<uint64_t*>(sw + TC_W_BYTES / 4);
    uint32_t* const taddr = reinterpret_cast<uint32_t*>(bar + 1);
    auto sa_buf = [&](int c) { return sm + (1 + c) * TC_WORDS; };
    constexpr int REM = LOGC - 5;
    const int R = rows;
    const int logM = logR + LOGC;
    const int groups = (R + nv - 1) / nv;
    const int per = groups * np;
    const int total = per * ninst;
    const int t = threadIdx.x;
    auto decode = [&](int gg, int& jj, int& uu, uint32_t*& A, const uint32_t*& B) {
        const int inst = gg / per;
        const int r = gg - inst * per;
        jj = r / groups;
        uu = (r - jj * groups) * nv;
        if (desc) { A = desc[inst].ra; B = A + ((size_t)np << logM); }
        else { A = ra; B = rb; }
        A += (size_t)jj << logM;
        B += (size_t)jj << logM;
    };

    int g = blockIdx.x;
    // the operand tiles need 1024-byte alignment, which dynamic shared memory
    // has here (the kernel has no static one)
    if (tc_smem(sm) & 1023u) {
        pdl_wait();   // the grid must not end before the kernel it follows
        if (t == 0) atomicOr(T.err, DEV_ERR_ALIGN);
        return;
    }
    if (t < 32) tc_alloc(tc_smem(taddr), TC_COLS);
    if (t == 0) tc_mbar_init(tc_smem(bar));
    pdl_wait();
    pdl_trigger();
    if (g < total) {
        int j, u0;
        uint32_t* A;
        const uint32_t* B;
        decode(g, j, u0, A, B);
        tc_prefetch<LOGC>(sa_buf(0), A, u0, nv, R);
        if (squaring != 1) tc_prefetch<LOGC>(sb, B, u0, nv, R);
        else cp_async_commit();
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tm = *taddr;
    // this warp's tile and lanes: thread t owns A row t, positions 32 t ..
    const uint32_t tl = tm + (uint32_t)((t >> 7) * 128) + ((uint32_t)(t & 96) << 16);
    const uint32_t bar_s = tc_smem(bar);
    uint32_t phase = 0;
    bool dead = false;
    // both tiles of a buffer through W; waits until the sums are in TMEM
    auto transform = [&](uint32_t* buf) {
        tc_fence_smem();
        tc_fence_before();
        __syncthreads();
        if (t == 0) {
            tc_fence_after();
            tc_mma_tile(tm, tc_smem(buf), tc_smem(sw));
            tc_mma_tile(tm + 128, tc_smem(buf) + TC_TILE_BYTES, tc_smem(sw));
            tc_commit(bar_s);
        }
        // a warp gives up as one, and is converged again (thread 0's branch, each
        // thread's own polls) before the aligned loads that follow
        if (!dead && !__all_sync(0xffffffffu, tc_mbar_wait(bar_s, phase))) {
            dead = true;                              // never on a working device: flag it and finish
            atomicOr(T.err, DEV_ERR_ROWS);
        }
        __syncwarp();
        phase ^= 1;
        tc_fence_after();
    };

    int cur = 0, jw = -1;
    for (; g < total; g += gridDim.x) {
        int j, u0, j2 = 0, u2 = 0;
        uint32_t *A, *A2 = nullptr;
        const uint32_t *B, *B2 = nullptr;
        decode(g, j, u0, A, B);
        const int g2 = g + gridDim.x;
        if (g2 < total) decode(g2, j2, u2, A2, B2);
        const PrimeInfo P = T.pi[j];
        const uint32_t p = P.p;
        const TcPrime K = T.tcp[j];
        const uint2* __restrict__ twf = T.twf + (size_t)j * TW_SZ;
        const uint2* __restrict__ twi = T.twi + (size_t)j * TW_SZ;
        uint32_t* sa = sa_buf(cur);

        if (j != jw) {
            // this prime's matrix (the last product with the old one has been waited for)
            const uint4* __restrict__ src = T.tcw + (size_t)j * (TC_W_BYTES / 16);
#pragma unroll
            for (int k = 0; k < TC_W_BYTES / 16 / TC_THREADS; k++)
                reinterpret_cast<uint4*>(sw)[t + k * TC_THREADS] = src[t + k * TC_THREADS];
            jw = j;
        }
        // this item's rows have landed; the other a buffer is free (its last
        // item stored from it before the barrier)
        cp_async_wait<0>();
        __syncthreads();
        if (g2 < total) tc_prefetch<LOGC>(sa_buf(cur ^ 1), A2, u2, nv, R);
        else cp_async_commit();

        uint32_t breg[32];
        if (squaring == 0) {
            // One pass of five levels: a vector at a time, and the instance still spills
            // (2^10-point rows: 236 bytes a thread; the other lengths none).  Two
            // vectors together would need twice the registers.
            if constexpr (REM == 5) {
                tc_gs_passes<LOGC, 1, 5, (1 << (LOGC - 1)), REM>(sb, sb, nv, twf, p);
                tc_gs_passes<LOGC, 1, 5, (1 << (LOGC - 1)), REM>(sa, sa, nv, twf, p);
            } else {
                tc_gs_passes<LOGC, 2, 5, (1 << (LOGC - 1)), REM>(sa, sb, nv, twf, p);
            }
            transform(sb);
#pragma unroll
            for (int i = 0; i < 4; i++) {
                uint32_t s[32];
                tc_ld32(s, tl + 32 * i);
#pragma unroll
                for (int m = 0; m < 8; m++)
                    breg[8 * i + m] = tc_reduce(s[4 * m], s[4 * m + 1], s[4 * m + 2], s[4 * m + 3], p, K);
            }
            // b's buffer has been read (its product is complete): refill it
            if (g2 < total) tc_prefetch<LOGC>(sb, B2, u2, nv, R);
            else cp_async_commit();
        } else {
            tc_gs_passes<LOGC, 1, 5, (1 << (LOGC - 1)), REM>(sa, sa, nv, twf, p);
            if (squaring == 2) {
                // b's rows already hold its spectrum in this kernel's order
#pragma unroll
                for (int q = 0; q < 8; q++) {
                    const uint4 v = *reinterpret_cast<const uint4*>(sb + 32 * t + 4 * (q ^ (t & 7)));
                    breg[4 * q] = v.x; breg[4 * q + 1] = v.y; breg[4 * q + 2] = v.z; breg[4 * q + 3] = v.w;
                }
                __syncthreads();   // b fully read: refill it for the next item
                if (g2 < total) tc_prefetch<LOGC>(sb, B2, u2, nv, R);
                else cp_async_commit();
            } else {
                cp_async_commit();
            }
        }
        transform(sa);
        const uint32_t sc = scale ? scale[j] : 0u;
        // a's spectrum, the pointwise product and this thread's row of the
        // inverse's operand: position bitrev5(m) takes output m, so the forward
        // matrix serves (its output m then has frequency bitrev5(m) of the
        // positions, the inverse's position -bitrev5(m) mod 32)
#pragma unroll
        for (int i = 0; i < 4; i++) {
            uint32_t s[32];
            tc_ld32(s, tl + 32 * i);
#pragma unroll
            for (int m = 0; m < 8; m++) {
                uint32_t x = tc_reduce(s[4 * m], s[4 * m + 1], s[4 * m + 2], s[4 * m + 3], p, K);
                x = red1(x, p);
                // one factor reduced: x y < 2 p^2, and the lazy Montgomery
                // product stays below 2 p < 2^32 (any 32-bit value may follow)
                const uint32_t y = squaring == 1 ? x : breg[8 * i + m];
                uint64_t w = (uint64_t)x * y;
                w += (uint64_t)((uint32_t)w * P.pneg_inv) * p;
                x = (uint32_t)(w >> 32);
                if (scale) x = mul_mont(red1(x, p), sc, p, P.pneg_inv);
                breg[8 * i + m] = x;
            }
        }
#pragma unroll
        for (int q = 0; q < 8; q++) {
            uint4 v;
            v.x = breg[__brev((unsigned)(4 * q)) >> 27];
            v.y = breg[__brev((unsigned)(4 * q + 1)) >> 27];
            v.z = breg[__brev((unsigned)(4 * q + 2)) >> 27];
            v.w = breg[__brev((unsigned)(4 * q + 3)) >> 27];
            *reinterpret_cast<uint4*>(sa + 32 * t + 4 * (q ^ (t & 7))) = v;
        }
        transform(sa);
#pragma unroll
        for (int i = 0; i < 4; i++) {
            uint32_t s[32];
            tc_ld32(s, tl + 32 * i);
#pragma unroll
            for (int m = 0; m < 8; m++)
                breg[8 * i + m] = red1(tc_reduce(s[4 * m], s[4 * m + 1], s[4 * m + 2], s[4 * m + 3], p, K), p);
        }
#pragma unroll
        for (int q = 0; q < 8; q++) {
            // position y is output m with bitrev5(m) = -y mod 32
            uint4 v;
            v.x = breg[__brev((unsigned)((32 - 4 * q) & 31)) >> 27];
            v.y = breg[__brev((unsigned)(31 - 4 * q)) >> 27];
            v.z = breg[__brev((unsigned)(30 - 4 * q)) >> 27];
            v.w = breg[__brev((unsigned)(29 - 4 * q)) >> 27];
            *reinterpret_cast<uint4*>(sa + 32 * t + 4 * (q ^ (t & 7))) = v;
        }
        __syncthreads();
        tc_ct_passes_out<LOGC, 5, 32, REM>(sa, nv, min(nv, R - u0), twi, p, A + ((size_t)u0 << LOGC));
        cur ^= 1;
    }
    cp_async_wait<0>();
    tc_fence_before();
    __syncthreads();
    if (t < 32) {
        tc_fence_after();
        tc_dealloc(tm, TC_COLS);
    }
}

}  // namespace fb
