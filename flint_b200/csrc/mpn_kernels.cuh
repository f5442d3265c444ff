// Kernels of the integer multiplication path z = a * b (mpn limbs, 64-bit).
//
// Coefficients are single limbs (64-bit chunks); the cyclic convolution of
// length M = 2^m = R * C is computed modulo np word-size primes with a
// four-step transform (C = 2^14 once M > 2^14, R = M / C <= 2^11):
//
//   k_fwd_cols   limbs -> residues (split fused into the load), length-R
//                forward transforms down G columns at a time, four-step twist
//                w_M^(i*k1) applied in registers, write.  [one pass over HBM]
//   k_rows       per row: forward transform of b (kept in registers), forward
//                transform of a, pointwise product with the CRT/normalisation
//                scale, inverse transform.               [one pass over HBM]
//   k_inv_cols   untwist in registers, length-R inverse transforms down the
//                columns.                                 [one pass over HBM]
//   k_crt_carry  np residues -> exact coefficient (CRT), coefficients ->
//                limbs with the carry chain resolved by a decoupled
//                look-back scan across tiles.             [one pass over HBM]
//
// Reference counterparts: limb splitting mpn_to_ffts_* (src/fft_small/
// mpn_mul.c:422-696), the per-prime transform/pointwise/inverse worker
// (mpn_mul.c:1505-1527), and CRT + carry recomposition _mpn_from_ffts_NP
// with the serial overhang stitch (mpn_mul.c:802-993, 1934-1973).
#pragma once
#include "ntt_smem.cuh"
#include "tcgen05.cuh"

namespace fb {

constexpr int LOG_MAXM = 25;              // largest cyclic length 2^25
constexpr int LOG_MAXC = 14;              // longest row transform
constexpr int TW_SZ = 1 << LOG_MAXC;      // local twiddle table entries per prime
constexpr int TH_SZ = 1 << (LOG_MAXM - 13);   // twist table: w^(t 2^13), t < 2^12
constexpr int TL_SZ = 1 << 13;            // twist table: w^t, t < 2^13

// Transforms of 3 2^k points (the first NP3 primes have roots of order
// 3 2^25): twist powers of w3 (order 3 2^25) and radix-3 stage twiddles
constexpr int NP3 = 5;
constexpr int TH3_SZ = 3 << (LOG_MAXM - 13);   // w3^(t 2^13), t < 3 2^12
constexpr int LOG_R3 = 11;                      // radix-3 stage tables serve columns up to 3 2^11
constexpr int TW3_SZ = 2 << LOG_R3;             // (omega^e / 2), e < 2^12, omega of order 3 2^11

struct DevTables {
    const PrimeInfo* pi;   // [MAX_NP]
    const uint2* twf;      // [MAX_NP][TW_SZ] forward local twiddles
    const uint2* twi;      // [MAX_NP][TW_SZ] inverse local twiddles
    const uint2* th;       // [MAX_NP][TH_SZ] w_{2^25}^(t 2^13)
    const uint2* tl;       // [MAX_NP][TL_SZ] w_{2^25}^t
    const uint2* thi;      // inverses of the above
    const uint2* tli;
    const uint2* th3;      // [NP3][TH3_SZ] w3^(t 2^13)
    const uint2* tl3;      // [NP3][TL_SZ] w3^t
    const uint2* th3i;     // inverses of the above
    const uint2* tl3i;
    const uint2* tw3f;     // [NP3][TW3_SZ] omega^e / 2, omega = w3^(2^14) of order 3 2^11
    const uint2* tw3i;     // [NP3][TW3_SZ] omega^-e / 2
    const uint2* w3c;      // [NP3][2] (w - w^2, w^-1 - w^-2), w = w3^(2^25) of order 3
    const uint4* tcw;      // [MAX_NP] swizzled W images (tc_fill_w), TC_W_BYTES each
    const TcPrime* tcp;    // [MAX_NP]
    int* err;              // the context's device error flag (DEV_ERR_*)
};

// Bits of a context's error flag, set by kernels whose results are not valid.
constexpr int DEV_ERR_CARRY = 1;   // a carry look-back gave up waiting
constexpr int DEV_ERR_ROWS = 2;    // the row pass gave up waiting for a matrix product
constexpr int DEV_ERR_ALIGN = 4;   // the row pass found its operand tiles misaligned

// Programmatic dependent launch.  A kernel launched as a programmatic
// dependent (launch_dep in lib.cu) may start while its predecessor on the
// stream still runs; pdl_wait() holds it until that predecessor has completed
// and its writes are visible, pdl_trigger() lets the successor start.  Without
// such a launch both do nothing.
// A short product is a chain of three or four kernels of 3-12 us each, so
// the launch gaps between them are a fifth of its time.  The forward column and
// the CRT kernels trigger just before their stores, not at their start: the
// row kernel's few CTAs, placed while all the column CTAs are still resident,
// share SMs that would be free a moment later (2^15 x 2^15 limbs: 30.1 us
// plain, 26.0 us with early triggers, 23.5 us with late ones; 2^11 x 2^11: 20.5,
// 25.0, 13.6 us).
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void pdl_trigger() { asm volatile("griddepcontrol.launch_dependents;"); }

// w_M^e * x for e in units of the largest transform (e < 2^25)
__device__ __forceinline__ uint32_t twist_mul(uint32_t x, uint32_t e, const uint2* __restrict__ th,
                                              const uint2* __restrict__ tl, uint32_t p)
{
    const uint2 w1 = th[e >> 13];
    const uint2 w2 = tl[e & 8191];
    x = mul_shoup(x, w1.x, w1.y, p);
    return mul_shoup(x, w2.x, w2.y, p);
}

__device__ __forceinline__ uint32_t bitrev_bits(uint32_t u, int bits)
{
    return bits == 0 ? 0u : (__brev(u) >> (32 - bits));
}

struct MulShape {
    int logR, logC;        // M = 2^(logR + logC)
    int G;                 // columns per column-pass tile
};

// columns per tile for a column length 2^logR: 32 KB tiles (256 threads; at 57 to 64
// registers four CTAs per SM, whose loads, levels and stores overlap -- the inverse
// pass of 2^5-point columns, whole in registers, takes 128 and two), at least 8
// columns (32-byte row segments).  Against 64 KB tiles of 512 threads, two per SM, which
// 2^11-point columns keep: columns of 2^8 points (2^20 x 2^20 limbs) forward 74.2 ->
// 68.3 us, inverse 36.6 -> 32.0; 2^9 137.7 -> 125.7, 61.6 -> 57.3; 2^10 284.0 ->
// 282.2, 135.0 -> 128.8.
__host__ __device__ constexpr int cols_per_tile(int logR)
{
    return logR >= 10 ? 8 : (1 << (13 - logR));
}

// w^e for e in units of the largest transform, from the two-level tables
__device__ __forceinline__ uint32_t table_power(uint32_t e, const uint2* __restrict__ th,
                                                const uint2* __restrict__ tl, uint32_t p)
{
    const uint2 w1 = th[e >> 13];
    const uint2 w2 = tl[e & 8191];
    return mul_shoup(w1.x, w2.x, w2.y, p);
}

// Shoup companion floor(w 2^32 / p) on the device: a double-precision
// estimate (error well below 1) corrected by one exact remainder test.
__device__ __forceinline__ uint32_t shoup_companion_dev(uint32_t w, uint32_t p)
{
    const double est = (double)w * (4294967296.0 / (double)p);
    uint32_t q = (uint32_t)est;
    const int64_t r = (int64_t)((uint64_t)w << 32) - (int64_t)((uint64_t)q * p);
    if (r >= (int64_t)p) q++;
    else if (r < 0) q--;
    return q;
}

// Four-step twist of the 32 consecutive column positions u = 32 s + m held by
// one thread: position u gets w_M^(col * bitrev_r(u)).  Since
// bitrev_r(32 s + m) = bitrev_(r-5)(s) + 2^(r-5) bitrev_5(m), the factors are
// alpha * beta^k, k = bitrev_5(m), with alpha = w^(col bitrev_(r-5)(s)) and
// beta = w^(col 2^(r-5)).  They are generated by a Shoup chain in Montgomery
// form (F_(k+1) = F_k beta) and applied with one Montgomery product each,
// so no table is read per element.
// fsc != 0 multiplies every factor by fsc (a pointwise scale folded into
// this operand's transform; one extra product per thread).
template <int LOGR>
__device__ __forceinline__ void twist32(uint32_t (&x)[32], uint32_t col, int s, int logM,
                                        const uint2* __restrict__ th, const uint2* __restrict__ tl,
                                        const PrimeInfo& P, uint32_t fsc = 0)
{
    const uint32_t p = P.p;
    const uint32_t mmask = (1u << logM) - 1;
    const int sh = LOG_MAXM - logM;
    const uint32_t e0 = ((col * bitrev_bits((uint32_t)s, LOGR - 5)) & mmask) << sh;
    const uint32_t e1 = ((col << (LOGR - 5)) & mmask) << sh;
    const uint32_t alpha = table_power(e0, th, tl, p);
    const uint32_t beta = table_power(e1, th, tl, p);
    const uint32_t bq = shoup_companion_dev(beta, p);
    uint32_t F = mul_mont(alpha, P.r2, p, P.pneg_inv);   // alpha in Montgomery form
    if (fsc) F = mul_mont(F, fsc, p, P.pneg_inv);         // alpha fsc, Montgomery form
#pragma unroll
    for (int k = 0; k < 32; k++) {
        const int m = (int)(__brev((unsigned)k) >> 27);
        x[m] = mul_mont(x[m], F, p, P.pneg_inv);
        if (k < 31) F = mul_shoup(F, beta, bq, p);
    }
}

// One product of a batch: operands, result, its residue scratch (a's np
// transforms at ra, b's at ra + np M) and its first CRT tile within the launch.
struct InstDesc {
    const uint64_t* a;
    const uint64_t* b;
    uint64_t* z;
    uint32_t* ra;
    uint64_t an, bn;
    uint32_t tile0, ntiles;
};

// Integer-polynomial operands: coefficient i of an operand is w 64-bit limbs
// in two's complement (the top limb signed), chunk k of it is placed at
// position i S + k of a polynomial in y (S = wa + wb - 1, so the chunk
// products of different output coefficients never share a position).
struct FzShape {
    uint32_t S;       // slot stride in y
    uint32_t wa, wb;  // limbs per coefficient of a and of b
};

// Residue (times 2^-32) of chunk k of coefficient i of an xn-coefficient
// polynomial with w limbs per coefficient (zero beyond the coefficient's
// limbs or the polynomial).
__device__ __forceinline__ uint32_t load_chunk(const uint64_t* __restrict__ x, uint32_t i, uint32_t k,
                                               uint64_t xn, uint32_t w, const PrimeInfo& P)
{
    if (k >= w || i >= xn) return 0u;
    const uint64_t v = x[(size_t)i * w + k];
    uint32_t r = limb_redc(v, P.p, P.pneg_inv, P.c32);
    // a negative top limb stands for v - 2^64, and 2^64 2^-32 = 2^32
    if (k == w - 1 && (int64_t)v < 0) r = sub_mod(r, P.c32, P.p);
    return r;
}

// Residue (times 2^-32) of operand element n.  Limb source: limb n of an
// xn-limb integer.  Coefficient source: chunk (n mod S) of coefficient n / S
// of an xn-coefficient polynomial with w limbs per coefficient.
template <bool FZ>
__device__ __forceinline__ uint32_t load_residue(const uint64_t* __restrict__ x, uint64_t n, uint64_t xn,
                                                 uint32_t S, uint32_t w, const PrimeInfo& P)
{
    if constexpr (!FZ) {
        return n < xn ? limb_redc(x[n], P.p, P.pneg_inv, P.c32) : 0u;
    } else {
        const uint32_t nn = (uint32_t)n;      // y-lengths stay below 2^32
        const uint32_t i = nn / S, k = nn - i * S;
        return load_chunk(x, i, k, xn, w, P);
    }
}

// Forward column instances that may run as programmatic dependents: short
// columns and narrow tiles, which only launches of a few CTAs per SM take.  The wide
// ones serve large products, where a launch gap is nothing and the wait's memory
// barrier costs the schedule of the loads (2^25-point forward pass 1.13 -> 1.5 ms
// with it compiled in).
template <int LOGR, int G>
__device__ __host__ constexpr bool fwd_cols_dep() { return LOGR < 5 || G < cols_per_tile(LOGR); }

// ---------------------------------------------------------------------------
// Column pass, forward: split + length-R transforms + twist.
// grid = (np, C / G, operands) -- the prime index varies fastest so that the
// np tiles that read the same limbs run together and share them through L2;
// with a batch descriptor, grid.z = 2 * instance + operand.  FZ selects the
// integer-polynomial source (an, bn count coefficients, shape in fz).
// smem = padw(R * G) words.
// LC != 0: the row length 2^LC is a compile-time constant (logC == LC), so
// the strided stores take immediate offsets instead of address arithmetic.
// DEP: the kernel may run as a programmatic dependent.
template <int LOGR, int G, bool FZ, int LC, bool DEP>
__device__ __forceinline__ void
fwd_cols_body(DevTables T, const uint64_t* __restrict__ a, uint64_t an,
              const uint64_t* __restrict__ b, uint64_t bn,
              uint32_t* __restrict__ ra, uint32_t* __restrict__ rb, int logC, int gcols,
              const InstDesc* __restrict__ desc, int np, FzShape fz, const uint32_t* __restrict__ fscale,
              int fmask)
{
    extern __shared__ uint32_t sm[];
    constexpr int R = 1 << LOGR;
    if constexpr (LC != 0) logC = LC;
    const int C = 1 << logC;
    const int logM = LOGR + logC;
    const int GR = G ? G : gcols;          // runtime tile width for short columns
    const int j = blockIdx.x;
    const int i0 = blockIdx.y * GR;
    const bool opb = (blockIdx.z & 1) != 0;
    if (desc) {
        const InstDesc& D = desc[blockIdx.z >> 1];
        a = D.a; b = D.b; an = D.an; bn = D.bn;
        ra = D.ra;
        rb = D.ra + ((size_t)np << logM);
    }
    const uint64_t* __restrict__ x = opb ? b : a;
    const uint64_t xn = opb ? bn : an;
    const uint32_t xw = opb ? fz.wb : fz.wa;
    uint32_t* __restrict__ out = (opb ? rb : ra) + ((size_t)j << logM);
    const PrimeInfo P = T.pi[j];
    const uint32_t p = P.p;
    const uint64_t M = (uint64_t)1 << logM;
    const int tot = R * GR;
    // threads of a tile with columns of 2^5 points or more: one per 32-point
    // column segment (256 for the 2^13-word tiles, 512 for 2^14, fewer for narrow ones)
    constexpr int NT = G ? (G * R / 32 < 512 ? G * R / 32 : 512) : 512;
    constexpr int PNT = NT + NT / 32;     // padw(NT)

    // Columns over 2^13-point rows run their first strided pass straight from the
    // limbs, without the tile's round trip through shared memory and one barrier:
    // 2^9-point columns 125.6 -> 121.1 us, 2^10 282.4 -> 268.6, 2^11 615 -> 578.
    // 2^14-point rows lost (1130 -> 1170 us) and shorter ones gained nothing; the
    // chunk loads of integer polynomials need a division per sub-transform.
    constexpr bool FUSED = !FZ && LC == 13;
    constexpr int Q1 = LOGR > 5 ? balanced_pass<(LOGR > 5 ? LOGR - 5 : 1), 4>() : 1;   // levels of the first strided pass
    bool first_done = false;
    if (FUSED && xn <= M) {
        // the first strided pass straight from the limbs: sub-transform s of
        // column v takes rows s + m S
        if constexpr (FUSED) {
            constexpr int E = 1 << Q1, S = R / E, GG = G ? G : 1;
            const uint2* __restrict__ tw = T.twf + (size_t)j * TW_SZ;
            constexpr int LS = LOGR - Q1;     // S = 2^LS rows
#pragma unroll 1
            for (int f = threadIdx.x; f < GG * S; f += NT) {
                const int v = f & (GG - 1), s = f / GG;
                const uint64_t n = ((uint64_t)s << logC) + i0 + v;
                int kin = 0;
                if (n < xn) {
                    const uint64_t q = ((xn - n - 1) >> (LS + logC)) + 1;
                    kin = q < (uint64_t)E ? (int)q : E;
                }
                const uint64_t* px = x + n;
                uint64_t lim[E];
#pragma unroll
                for (int m = 0; m < E; m++) lim[m] = m < kin ? px[(size_t)m << (LS + logC)] : 0ull;
                uint32_t xr[E];
#pragma unroll
                for (int m = 0; m < E; m++) xr[m] = limb_redc(lim[m], p, P.pneg_inv, P.c32);
                gs_strided<Q1, R / 2, COL_FMA_ADDS>(xr, tw, s, p);
                uint32_t* d = sm + padw(s * GG) + v;
#pragma unroll
                for (int m = 0; m < E; m++) d[padw(m * S * GG)] = xr[m];
            }
            first_done = true;
        }
    } else if (LOGR >= 5 && (FZ || xn <= M)) {
        // blockDim == G R / 32 == NT: thread t loads elements t + NT k, i.e.
        // rows u_t + k NT/G of its fixed column; shared offsets are constants
        const int t = threadIdx.x;
        const int GG = G ? G : 1;
        const int u_t = t / GG, c = t & (GG - 1);
        const uint64_t step = (uint64_t)(NT / GG) * C;
        uint64_t n = (uint64_t)u_t * C + i0 + c;
        uint32_t* d = sm + padw(u_t * GG) + c;
        if constexpr (!FZ && LOGR >= 5) {
            // step is a power of two: the number of loads inside the operand
            // is a shift, and a pointer bump per row keeps the 64-bit address
            // arithmetic off the FMA pipe (measured 1.267 -> 1.249 ms for the
            // two operands of a 2^24 x 2^24 product)
            constexpr int K = R * GG / NT;
            const int lstep = (31 - __clz(NT / GG)) + logC;
            int kin = 0;
            if (n < xn) {
                const uint64_t q = ((xn - n - 1) >> lstep) + 1;
                kin = q < (uint64_t)K ? (int)q : K;
            }
            const uint64_t* px = x + n;
#pragma unroll 8
            for (int k = 0; k < K; k++, px += step)
                d[k * PNT] = k < kin ? limb_redc(*px, p, P.pneg_inv, P.c32) : 0u;
        } else if constexpr (FZ) {
            // integer-polynomial source: n advances by `step`, so its slot
            // n / S and chunk n mod S advance by fixed amounts (one division
            // per thread instead of one per element)
            const uint32_t S = fz.S;
            uint32_t ci = (uint32_t)n / S, ck = (uint32_t)n - ci * S;
            const uint32_t sq = (uint32_t)step / S, sr = (uint32_t)step - sq * S;
            // the limb offset ci w + ck advances the same way
            size_t off = (size_t)ci * xw + ck;
            const size_t doff = (size_t)sq * xw + sr;
#pragma unroll 8
            for (int k = 0; k < R * GG / NT; k++) {
                uint32_t r = 0;
                if (ck < xw && ci < xn) {
                    const uint64_t v = x[off];
                    r = limb_redc(v, p, P.pneg_inv, P.c32);
                    // a negative top limb stands for v - 2^64
                    if (ck == xw - 1 && (int64_t)v < 0) r = sub_mod(r, P.c32, p);
                }
                d[k * PNT] = r;
                ci += sq;
                ck += sr;
                off += doff;
                if (ck >= S) {
                    ck -= S;
                    ci++;
                    off -= (size_t)(S - xw);   // S >= xw: one slot on, minus the chunks it carries
                }
            }
        } else {
#pragma unroll 8
            for (int k = 0; k < R * GG / NT; k++, n += step)
                d[k * PNT] = load_residue<FZ>(x, n, xn, fz.S, xw, P);
        }
    } else if (FZ || xn <= M) {
        // four loads in flight per thread (small transforms are bound by
        // their latency)
        for (int f0 = threadIdx.x; f0 < tot; f0 += 4 * blockDim.x) {
            uint32_t v[4];
#pragma unroll
            for (int q = 0; q < 4; q++) {
                const int f = f0 + q * (int)blockDim.x;
                const int u = f / GR, c = f - u * GR;
                v[q] = f < tot ? load_residue<FZ>(x, (uint64_t)u * C + i0 + c, xn, fz.S, xw, P) : 0u;
            }
#pragma unroll
            for (int q = 0; q < 4; q++) {
                const int f = f0 + q * (int)blockDim.x;
                const int u = f / GR, c = f - u * GR;
                if (f < tot) sm[padw(u * GR) + c] = v[q];
            }
        }
    } else {
        // cyclic fold: an operand longer than M wraps around (x mod X^M - 1)
        for (int f = threadIdx.x; f < tot; f += blockDim.x) {
            const int u = f / GR, c = f - u * GR;
            uint32_t r = 0;
            for (uint64_t n = (uint64_t)u * C + i0 + c; n < xn; n += M)
                r = add_mod(r, limb_redc(x[n], p, P.pneg_inv, P.c32), p);
            sm[padw(u * GR) + c] = r;
        }
    }
    __syncthreads();
    const uint2* __restrict__ th = T.th + (size_t)j * TH_SZ;
    const uint2* __restrict__ tl = T.tl + (size_t)j * TL_SZ;
    const int sh = LOG_MAXM - logM;
    const uint32_t mmask = (uint32_t)(M - 1);
    if constexpr (LOGR >= 5) {
        // pointwise scale folded into this operand's twist (fmask bit 0: the
        // first operand, bit 1: the second)
        const uint32_t fsc = (fmask >> (opb ? 1 : 0)) & 1 ? fscale[j] : 0u;
        if constexpr (FUSED) {
            if (!first_done) {
                gs_pass_smem<LOGR, Q1, R / 2, G>(sm, 1, T.twf + (size_t)j * TW_SZ, p);
                __syncthreads();
            }
            gs_passes<LOGR, G, 4, ((R / 2) >> Q1), LOGR - 5 - Q1>(sm, 1, T.twf + (size_t)j * TW_SZ, p);
        } else {
            gs_strided_all<LOGR, G>(sm, 1, T.twf + (size_t)j * TW_SZ, p);
        }
        constexpr int NS = R / 32;
        for (int f = threadIdx.x; f < G * NS; f += blockDim.x) {
            const int v = f & (G - 1), s = f / G;
            const int pb = 33 * G * s + v;
            uint32_t xr[32];
#pragma unroll
            for (int m = 0; m < 32; m++) xr[m] = sm[pb + padw(m * G)];
            gs_contig<5, COL_FMA_ADDS>(xr, c_w32[j], p);
            const uint32_t col = (uint32_t)(i0 + v);
            twist32<LOGR>(xr, col, s, logM, th, tl, P, fsc);
            if constexpr (DEP) pdl_trigger();
            // rows 32 s .. 32 s + 31 of column col: a pointer bump per row keeps
            // the address arithmetic on the ALU pipe (the FMA pipe is this
            // kernel's busiest unit)
            uint32_t* o = out + ((size_t)(32 * s) << logC) + col;
            if constexpr (LC != 0) {
#pragma unroll
                for (int m = 0; m < 32; m++) o[m * (1 << LC)] = xr[m];
            } else {
#pragma unroll
                for (int m = 0; m < 32; m++, o += C) *o = xr[m];
            }
        }
    } else {
        // short columns: one thread owns a whole column
        for (int v = threadIdx.x; v < GR; v += blockDim.x) {
            uint32_t xr[R];
#pragma unroll
            for (int m = 0; m < R; m++) xr[m] = sm[padw(m * GR) + v];
            if constexpr (LOGR > 0) gs_contig<LOGR, COL_FMA_ADDS>(xr, c_w32[j], p);
            const uint32_t col = (uint32_t)(i0 + v);
#pragma unroll
            for (int m = 0; m < R; m++) {
                uint32_t val = xr[m];
                if constexpr (LOGR > 0) {
                    const uint32_t e = ((col * bitrev_bits(m, LOGR)) & mmask) << sh;
                    val = twist_mul(val, e, th, tl, p);
                }
                out[(size_t)m * C + col] = val;
            }
        }
    }
}

// Kernel instances: LC = 0 takes the row length at run time; LC = 14 serves
// 2^14-point rows under 2^11-point columns (2^25 points) and LC = 13 2^13-point
// rows under 2^9- to 2^11-point columns, with constant strides (measured on
// the 2^25-point forward pass: 1.28 -> 1.13 ms).  An LC instance also holds
// the run-time body behind a branch that never takes it for its shape: with
// that second body the compiler schedules the constant-stride one better
// (1.21 ms alone, 1.13 ms with it; three bodies in one kernel: 1.24 ms).
template <int LOGR, int G, bool FZ, int LC = 0, bool DEP = fwd_cols_dep<LOGR, G>()>
__global__ void __launch_bounds__(512)
k_fwd_cols(DevTables T, const uint64_t* __restrict__ a, uint64_t an,
           const uint64_t* __restrict__ b, uint64_t bn,
           uint32_t* __restrict__ ra, uint32_t* __restrict__ rb, int logC, int gcols,
           const InstDesc* __restrict__ desc, int np, FzShape fz, const uint32_t* __restrict__ fscale,
           int fmask)
{
    if constexpr (DEP) pdl_wait();
    if (LC != 0 && logC == LC)
        fwd_cols_body<LOGR, G, FZ, LC, DEP>(T, a, an, b, bn, ra, rb, logC, gcols, desc, np, fz, fscale, fmask);
    else
        fwd_cols_body<LOGR, G, FZ, 0, DEP>(T, a, an, b, bn, ra, rb, logC, gcols, desc, np, fz, fscale, fmask);
}

// ---------------------------------------------------------------------------
// Row pass, persistent: each CTA walks over items of nv rows (one prime per
// item).  For every item: forward transforms of a and b as one interleaved
// network (shared twiddle loads, twice the independent work per thread; b's
// spectrum ends in registers), pointwise product times scale[j], inverse
// transform; the result overwrites the a rows.  Three shared buffers: b, and
// a ping-pong pair for a, so the next item's a rows stream in (cp.async)
// during the whole current item and its b rows as soon as b's spectrum is in
// registers.  grid = min(items, resident CTAs); block = nv * C / 32;
// smem = 3 * nv * padw(C) words.  `squaring`: 0 a b, 1 a a (b unused), 2 a
// times a b whose rows already hold its spectrum in this kernel's order
// (k_rows_fwd output; the chunks of a split product share one).
__device__ __forceinline__ void cp_async4(uint32_t* dst, const uint32_t* src, bool valid)
{
    const unsigned s = (unsigned)__cvta_generic_to_shared(dst);
    const int n = valid ? 4 : 0;   // a zero source size fills the word with zeros
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;\n" ::"r"(s), "l"(src), "r"(n));
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::); }
template <int N>
__device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;\n" ::"n"(N)); }

__device__ __forceinline__ void cp_async4_full(uint32_t* dst, const uint32_t* src)
{
    const unsigned s = (unsigned)__cvta_generic_to_shared(dst);
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;\n" ::"r"(s), "l"(src));
}

// 16 bytes, both addresses 16-byte aligned; bypasses L1 (.cg)
__device__ __forceinline__ void cp_async16(uint32_t* dst, const uint32_t* src)
{
    const unsigned s = (unsigned)__cvta_generic_to_shared(dst);
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(s), "l"(src));
}

// LOGE: log2 of the elements each thread owns in the row kernel's
// contiguous pass (blockDim = nv C / 2^LOGE).  UNP: a single row (nv = 1,
// rows of at least 2^10 words) lands unpadded, as 16-byte copies that bypass
// L1 -- 4x fewer copy instructions than the padded layout's 4-byte ones and
// no L1 allocation; the first forward pass pads it (gs_pass_first_unpadded).
// The row base and dst must be 16-byte aligned (residue planes and rows are
// multiples of 2^10 words; dst is a row buffer at a multiple of padw(C)).
template <int LOGC, int LOGE = 5>
__device__ __forceinline__ constexpr bool rows_unpadded(int nv)
{
    return LOGE == 5 && LOGC >= 10 && nv == 1;
}

template <int LOGC, int LOGE = 5, bool UNP = false>
__device__ __forceinline__ void rows_prefetch(uint32_t* dst, const uint32_t* __restrict__ base,
                                              int u0, int nv, int R)
{
    constexpr int C = 1 << LOGC;
    constexpr int PC = padw(C);
    constexpr int NSUB = C >> LOGE;
    if (UNP && rows_unpadded<LOGC, LOGE>(nv)) {
        // blockDim == NSUB == C / 32: 16-byte chunk c = t + k NSUB, k < 8
        const uint32_t* src = base + (size_t)u0 * C;
#pragma unroll
        for (int k = 0; k < (1 << LOGE) / 4; k++) {
            const int c = threadIdx.x + k * NSUB;
            cp_async16(dst + 4 * c, src + 4 * c);
        }
    } else if (nv == 1 && NSUB % 32 == 0) {
        // one row, blockDim == NSUB: element t + k NSUB, compile-time offsets
        const int t = threadIdx.x;
        const uint32_t* src = base + (size_t)u0 * C + t;
        uint32_t* d = dst + padw(t);
#pragma unroll
        for (int k = 0; k < (1 << LOGE); k++) cp_async4_full(d + k * (NSUB / 32 * 33), src + k * NSUB);
    } else {
        for (int f = threadIdx.x; f < nv * C; f += blockDim.x) {
            const int v = f >> LOGC, i = f & (C - 1);
            const int u = u0 + v;
            cp_async4(&dst[v * PC + padw(i)], base + (size_t)min(u, R - 1) * C + i, u < R);
        }
    }
    cp_async_commit();
}

// 2^14-point rows at 32 points per thread run large products only, which gain
// nothing from an early launch (1.474 ms; 1.483 ms with the wait compiled in).
template <int LOGC, int LOGE>
__device__ __host__ constexpr bool rows_dep() { return LOGC < LOG_MAXC || LOGE < 5; }

template <int LOGC, int LOGE = 5>
__global__ void __launch_bounds__(LOGE < 5 ? 1024 : 512, 1)
k_rows(DevTables T, uint32_t* __restrict__ ra, const uint32_t* __restrict__ rb,
       int logR, int nv, int np, const uint32_t* __restrict__ scale, int squaring,
       const InstDesc* __restrict__ desc, int ninst, int rows)
{
    extern __shared__ __align__(16) uint32_t sm[];   // 16-byte copies land in the row buffers
    constexpr int C = 1 << LOGC;
    constexpr int PC = padw(C);
    constexpr int E = 1 << LOGE;          // elements per thread in the contiguous pass
    constexpr int NSUB = C / E;
    constexpr int QMAX = LOGE;            // strided passes: at least one sub-transform per thread
    const int R = rows;                    // rows per prime (<= 2^logR, the prime stride's rows)
    const int logM = logR + LOGC;
    const int groups = (R + nv - 1) / nv;
    const int per = groups * np;           // items of one product
    const int total = per * ninst;
    uint32_t* sb = sm;
    // a ping-pong pair at sm + nv PC and sm + 2 nv PC (pointer arithmetic, not
    // an indexed array, so nothing goes to local memory)
    auto sa_buf = [&](int c) { return sm + (1 + c) * nv * PC; };
    const int t = threadIdx.x;
    const int pb = (t / NSUB) * PC + padw(E * (t & (NSUB - 1)));
    // item -> (prime, first row, residue base of a, of b)
    auto decode = [&](int gg, int& jj, int& uu, uint32_t*& A, const uint32_t*& B) {
        const int inst = gg / per;
        const int r = gg - inst * per;
        jj = r / groups;
        uu = (r - jj * groups) * nv;
        if (desc) { A = desc[inst].ra; B = A + ((size_t)np << logM); }
        else { A = ra; B = rb; }
    };

    int g = blockIdx.x;
    if constexpr (rows_dep<LOGC, LOGE>()) {
        pdl_wait();
        pdl_trigger();
    }
    if (g >= total) return;
    {
        int j, u0;
        uint32_t* A;
        const uint32_t* B;
        decode(g, j, u0, A, B);
        rows_prefetch<LOGC, LOGE, true>(sa_buf(0), A + ((size_t)j << logM), u0, nv, R);
        if (squaring == 0) rows_prefetch<LOGC, LOGE, true>(sb, B + ((size_t)j << logM), u0, nv, R);
        else if (squaring == 2) rows_prefetch<LOGC, LOGE, false>(sb, B + ((size_t)j << logM), u0, nv, R);
        else cp_async_commit();
    }
    int cur = 0;
    for (; g < total; g += gridDim.x) {
        int j, u0, j2 = 0, u2 = 0;
        uint32_t *A, *A2 = nullptr;
        const uint32_t *B, *B2 = nullptr;
        decode(g, j, u0, A, B);
        const int g2 = g + gridDim.x;
        if (g2 < total) decode(g2, j2, u2, A2, B2);
        const PrimeInfo P = T.pi[j];
        const uint32_t p = P.p;
        const uint2* __restrict__ twf = T.twf + (size_t)j * TW_SZ;
        const uint2* __restrict__ twi = T.twi + (size_t)j * TW_SZ;
        uint32_t* sa = sa_buf(cur);

        // this item's a and b rows have landed; the other a buffer is free
        // (its last item stored from it before the barrier)
        cp_async_wait<0>();
        __syncthreads();
        if (g2 < total) rows_prefetch<LOGC, LOGE, true>(sa_buf(cur ^ 1), A2 + ((size_t)j2 << logM), u2, nv, R);
        else cp_async_commit();

        uint32_t xr[E];
        uint32_t breg[E];
        if (squaring == 0) {
            if constexpr (LOGE == 5) {
                if (rows_unpadded<LOGC, LOGE>(nv)) gs_strided_all2<LOGC, QMAX, LOGE, true>(sa, sb, nv, twf, p);
                else gs_strided_all2<LOGC, QMAX, LOGE>(sa, sb, nv, twf, p);
            } else {
                gs_strided_all2<LOGC, QMAX, LOGE>(sa, sb, nv, twf, p);
            }
#pragma unroll
            for (int m = 0; m < E; m++) {
                xr[m] = sa[pb + m];
                breg[m] = sb[pb + m];
            }
            gs_contig2<LOGE, ROW_GS_FMA_ADDS>(xr, breg, c_w32[j], p);
            __syncthreads();   // b fully read: refill it for the next item
            if (g2 < total) rows_prefetch<LOGC, LOGE, true>(sb, B2 + ((size_t)j2 << logM), u2, nv, R);
            else cp_async_commit();
        } else {
            // a squaring, or b's rows already hold its spectrum in this
            // kernel's order (squaring == 2: k_rows_fwd output, landed padded)
            if constexpr (LOGE == 5) {
                if (rows_unpadded<LOGC, LOGE>(nv)) gs_strided_all<LOGC, 0, QMAX, LOGE, true>(sa, nv, twf, p);
                else gs_strided_all<LOGC, 0, QMAX, LOGE>(sa, nv, twf, p);
            } else {
                gs_strided_all<LOGC, 0, QMAX, LOGE>(sa, nv, twf, p);
            }
#pragma unroll
            for (int m = 0; m < E; m++) xr[m] = sa[pb + m];
            gs_contig<LOGE, ROW_GS_FMA_ADDS>(xr, c_w32[j], p);
            if (squaring == 2) {
#pragma unroll
                for (int m = 0; m < E; m++) breg[m] = sb[pb + m];
                __syncthreads();   // b fully read: refill it for the next item
                if (g2 < total) rows_prefetch<LOGC, LOGE, false>(sb, B2 + ((size_t)j2 << logM), u2, nv, R);
                else cp_async_commit();
            } else {
                cp_async_commit();
            }
        }
        if (scale) {
            const uint32_t sc = scale[j];
#pragma unroll
            for (int m = 0; m < E; m++) {
                const uint32_t y = squaring == 1 ? xr[m] : breg[m];
                xr[m] = mul_mont(mul_mont(xr[m], y, p, P.pneg_inv), sc, p, P.pneg_inv);
            }
        } else {
            // the scale was folded into a column pass (or a ring product's untwist)
#pragma unroll
            for (int m = 0; m < E; m++) xr[m] = mul_mont(xr[m], squaring == 1 ? xr[m] : breg[m], p, P.pneg_inv);
        }
        ct_contig<LOGE, ROW_CT_FMA_ADDS>(xr, c_w32[j], p);
#pragma unroll
        for (int m = 0; m < E; m++) sa[pb + m] = xr[m];
        __syncthreads();
        uint32_t* __restrict__ abase = A + ((size_t)j << logM);
        if constexpr (LOGC > LOGE) {
            if (nv == 1) {
                // one row: the last inverse pass writes it to HBM directly
                ct_strided_all_out<LOGC, QMAX, LOGE>(sa, twi, p, abase + (size_t)u0 * C);
                cur ^= 1;
                continue;
            }
        }
        ct_strided_all<LOGC, 0, QMAX, LOGE>(sa, nv, twi, p);
        if (nv == 1 && NSUB % 32 == 0) {
            uint32_t* dst = abase + (size_t)u0 * C + t;
            const uint32_t* s_ = sa + padw(t);
#pragma unroll
            for (int k = 0; k < E; k++) dst[k * NSUB] = s_[k * (NSUB / 32 * 33)];
        } else {
            for (int f = t; f < nv * C; f += blockDim.x) {
                const int v = f >> LOGC, i = f & (C - 1);
                const int u = u0 + v;
                if (u < R) abase[(size_t)u * C + i] = sa[v * PC + padw(i)];
            }
        }
        cur ^= 1;
    }
    cp_async_wait<0>();
}

// ---------------------------------------------------------------------------
// Transforms of one row (M = 2^LOGC points, no columns) in one launch: split,
// forward transforms of a and b, pointwise product, inverse transform.  One CTA
// per (prime, product), C / 2^LOGE threads; grid = (np, instances), smem =
// 2 padw(C) words; arguments as k_fwd_cols and k_rows.  A product of this
// length is bound by latency: launches, and instructions that every warp runs
// once from a cold cache.  Eight words per thread halve a warp's instructions
// against sixteen (256 x 256 limbs: 10.4 us with the split as a launch of its own,
// 11.4 us here with sixteen words per thread, 7.9 us with eight; 2048 x 2048:
// 13.2, 15.7, 13.0); a batch with enough products is bound by their number and
// takes sixteen (2^11 points 0.31 us a product with the split apart, 0.16 here,
// 0.18 with eight).
template <int LOGC, bool FZ, int LOGE>
__global__ void __launch_bounds__(1 << (LOGC - LOGE))
k_rows_small(DevTables T, const uint64_t* __restrict__ a, uint64_t an, const uint64_t* __restrict__ b, uint64_t bn,
             uint32_t* __restrict__ ra, const uint32_t* __restrict__ scale, int squaring,
             const InstDesc* __restrict__ desc, FzShape fz)
{
    extern __shared__ uint32_t sm[];
    constexpr int C = 1 << LOGC, E = 1 << LOGE, NT = C / E;
    static_assert(NT % 32 == 0, "whole warps");
    const int t = threadIdx.x, j = blockIdx.x;
    pdl_wait();
    pdl_trigger();
    if (desc) {
        const InstDesc& D = desc[blockIdx.y];
        a = D.a; b = D.b; an = D.an; bn = D.bn;
        ra = D.ra;
    }
    const PrimeInfo P = T.pi[j];
    const uint32_t p = P.p;
    uint32_t* const sa = sm;
    uint32_t* const sb = sm + padw(C);
    auto split = [&](uint32_t* s, const uint64_t* __restrict__ x, uint64_t xn, uint32_t xw) {
        if (FZ || xn <= (uint64_t)C) {
#pragma unroll
            for (int k = 0; k < E; k++)
                s[padw(t) + k * (NT / 32 * 33)] = load_residue<FZ>(x, (uint64_t)(t + k * NT), xn, fz.S, xw, P);
        } else {
            // an operand longer than the transform wraps around (x mod X^C - 1)
            for (int k = 0; k < E; k++) {
                uint32_t r = 0;
                for (uint64_t n = (uint64_t)(t + k * NT); n < xn; n += C)
                    r = add_mod(r, limb_redc(x[n], p, P.pneg_inv, P.c32), p);
                s[padw(t) + k * (NT / 32 * 33)] = r;
            }
        }
    };
    split(sa, a, an, fz.wa);
    if (!squaring) split(sb, b, bn, fz.wb);
    __syncthreads();
    const uint2* __restrict__ twf = T.twf + (size_t)j * TW_SZ;
    const uint2* __restrict__ twi = T.twi + (size_t)j * TW_SZ;
    const int pb = padw(E * t);
    uint32_t xr[E], br[E];
    if (!squaring) {
        gs_strided_all2<LOGC, LOGE, LOGE>(sa, sb, 1, twf, p);
#pragma unroll
        for (int m = 0; m < E; m++) {
            xr[m] = sa[pb + m];
            br[m] = sb[pb + m];
        }
        gs_contig2<LOGE, ROW_GS_FMA_ADDS>(xr, br, c_w32[j], p);
    } else {
        gs_strided_all<LOGC, 0, LOGE, LOGE>(sa, 1, twf, p);
#pragma unroll
        for (int m = 0; m < E; m++) xr[m] = sa[pb + m];
        gs_contig<LOGE, ROW_GS_FMA_ADDS>(xr, c_w32[j], p);
    }
    const uint32_t sc = scale[j];
#pragma unroll
    for (int m = 0; m < E; m++) {
        const uint32_t y = squaring ? xr[m] : br[m];
        xr[m] = mul_mont(mul_mont(xr[m], y, p, P.pneg_inv), sc, p, P.pneg_inv);
    }
    ct_contig<LOGE, ROW_CT_FMA_ADDS>(xr, c_w32[j], p);
#pragma unroll
    for (int m = 0; m < E; m++) sa[pb + m] = xr[m];
    __syncthreads();
    ct_strided_all_out<LOGC, LOGE, LOGE>(sa, twi, p, ra + ((size_t)j << LOGC));
}

// Destination of one chunk of a split product (a long operand cut into
// chunks, each multiplied by the short one): the inverse column pass writes
// the chunk's residues into acc (prime stride 2^logMf) at offset shift
// instead of back in place, adds them mod p below `overlap` (where the
// previous chunk's product ends), and skips positions at or beyond nvalid
// (past the chunk's product).  acc == nullptr: in place.
struct ChunkOut {
    uint32_t* acc;
    int logMf;
    uint64_t shift, overlap, nvalid;
};

// ---------------------------------------------------------------------------
// Column pass, inverse: untwist in registers + length-R inverse transforms,
// in place (or into a split product's residues, ChunkOut).  grid = (C / G, np, instances); smem = padw(R * G) words.
// SC: the pointwise scale folded into the untwist (squarings; as instances of
// their own, since the run-time choice cost the others 6%: 2^10-point columns
// 120.8 -> 128.3 us).
template <int LOGR, int G, int LC, bool SC>
__device__ __forceinline__ void
inv_cols_body(DevTables T, uint32_t* __restrict__ ra, int logC, int gcols,
              const InstDesc* __restrict__ desc, ChunkOut co, const uint32_t* __restrict__ fscale)
{
    extern __shared__ uint32_t sm[];
    constexpr int R = 1 << LOGR;
    if constexpr (LC != 0) logC = LC;
    const int C = 1 << logC;
    const int logM = LOGR + logC;
    const int GR = G ? G : gcols;
    const int j = blockIdx.y;
    uint32_t fsc = 0;
    if constexpr (SC) fsc = fscale[j];
    const int i0 = blockIdx.x * GR;
    if (desc) ra = desc[blockIdx.z].ra;
    uint32_t* __restrict__ buf = ra + ((size_t)j << logM);
    const PrimeInfo P = T.pi[j];
    const uint32_t p = P.p;
    const uint2* __restrict__ th = T.thi + (size_t)j * TH_SZ;
    const uint2* __restrict__ tl = T.tli + (size_t)j * TL_SZ;
    const int sh = LOG_MAXM - logM;
    const uint32_t mmask = (uint32_t)(((uint64_t)1 << logM) - 1);

    if constexpr (LOGR >= 5) {
        // element u of column v of a split product's chunk
        auto chunk_store = [&](int u, int v, uint32_t x) {
            uint32_t* __restrict__ out = co.acc + ((size_t)j << co.logMf) + co.shift;
            const uint64_t n = (uint64_t)u * C + i0 + v;
            if (n < co.nvalid) out[n] = n < co.overlap ? add_mod(out[n], x, p) : x;
        };
        constexpr int NS = R / 32;
        for (int f = threadIdx.x; f < G * NS; f += blockDim.x) {
            const int v = f & (G - 1), s = f / G;
            const uint32_t col = (uint32_t)(i0 + v);
            uint32_t xr[32];
            const uint32_t* src = buf + ((size_t)(32 * s) << logC) + col;
#pragma unroll
            for (int m = 0; m < 32; m++) xr[m] = src[(size_t)m * C];
            twist32<LOGR>(xr, col, s, logM, th, tl, P, fsc);
            ct_contig<5, COL_CT_FMA_ADDS>(xr, c_w32[j], p);
            if constexpr (LOGR == 5) {
                // the whole column is in registers
                if (!co.acc) {
                    uint32_t* dst = buf + col;
#pragma unroll
                    for (int m = 0; m < 32; m++) dst[(size_t)m * C] = xr[m];
                } else {
#pragma unroll
                    for (int m = 0; m < 32; m++) chunk_store(m, v, xr[m]);
                }
            } else {
                const int pb = 33 * G * s + v;
#pragma unroll
                for (int m = 0; m < 32; m++) sm[pb + padw(m * G)] = xr[m];
            }
        }
        if constexpr (LOGR > 5) {
            __syncthreads();
            // the last strided pass stores from registers: the tile's way back
            // through shared memory and its barrier cost columns of 2^10 points
            // 127.8 us against 120.8, of 2^9 57.4 against 53.7 (2^11: even)
            const uint2* __restrict__ twi = T.twi + (size_t)j * TW_SZ;
            if (!co.acc) {
                uint32_t* dst = buf + i0;
                ct_passes_cols_out<LOGR, G, 4, 32, LOGR - 5>(sm, twi, p, [&](int u, int v, uint32_t x) {
                    dst[(size_t)u * C + v] = x;
                });
            } else {
                ct_passes_cols_out<LOGR, G, 4, 32, LOGR - 5>(sm, twi, p, chunk_store);
            }
        }
    } else if constexpr (LOGR > 0) {
        for (int v = threadIdx.x; v < GR; v += blockDim.x) {
            const uint32_t col = (uint32_t)(i0 + v);
            uint32_t xr[R];
#pragma unroll
            for (int m = 0; m < R; m++) {
                const uint32_t e = ((col * bitrev_bits(m, LOGR)) & mmask) << sh;
                xr[m] = twist_mul(buf[(size_t)m * C + col], e, th, tl, p);
            }
            ct_contig<LOGR, COL_CT_FMA_ADDS>(xr, c_w32[j], p);
#pragma unroll
            for (int m = 0; m < R; m++) buf[(size_t)m * C + col] = xr[m];
        }
    }
}

template <int LOGR, int G, int LC = 0, bool SC = false>
__global__ void __launch_bounds__(512)
k_inv_cols(DevTables T, uint32_t* __restrict__ ra, int logC, int gcols,
           const InstDesc* __restrict__ desc, ChunkOut co, const uint32_t* __restrict__ fscale)
{
    // as the forward pass: the constant-stride instances serve large products
    if constexpr (LC == 0) {
        pdl_wait();
        pdl_trigger();
    }
    inv_cols_body<LOGR, G, LC, SC>(T, ra, logC, gcols, desc, co, fscale);
}

// ---------------------------------------------------------------------------
// CRT + carry.
//
// The inverse transforms leave y_j = (h mod p_j) * (P/p_j)^-1 mod p_j for each
// coefficient h of the product (the factor was folded into the pointwise
// scale).  Then h = sum_j y_j (P/p_j) - k P with k = round(sum_j y_j / p_j):
// the coefficient bound guarantees h < P/2, so the fractional part of
// sum_j y_j / p_j is h / P < 1/2 and the float estimate rounds to k exactly.
struct CrtConst {
    int np;
    uint32_t P[MAX_NP];               // product of the primes, 32-bit words
    uint32_t cof[MAX_NP][MAX_NP];     // P / p_j, 32-bit words
    float finv[MAX_NP];
    uint32_t Pneg[MAX_NP];            // 2^(32 np) - P, np words
    float kc[MAX_NP], koff;           // 2^8 / p_j; -2^23 sum_j kc[j]
};

template <int NP>
__device__ __forceinline__ void crt_values(const uint32_t (&y)[NP], const CrtConst& K, uint64_t& c0,
                                           uint64_t& c1, uint64_t& c2);

template <int NP>
__device__ __forceinline__ void crt_coeff(const uint32_t* __restrict__ res, int logM, uint64_t n,
                                          const CrtConst& K, uint64_t& c0, uint64_t& c1, uint64_t& c2)
{
    if constexpr (NP == 0) {
        // direct values: three word planes of L words each (L = 2^logM here)
        const uint64_t* v = reinterpret_cast<const uint64_t*>(res);
        const size_t L = (size_t)1 << logM;
        c0 = v[n]; c1 = v[L + n]; c2 = v[2 * L + n];
    } else {
        uint32_t y[NP];
#pragma unroll
        for (int jp = 0; jp < NP; jp++) y[jp] = res[((size_t)jp << logM) + n];
        crt_values<NP>(y, K, c0, c1, c2);
    }
}

// (a0 .. a3, a4) += (b0, b1) as 64-bit pairs, with the carry into a4
__device__ __forceinline__ void add128c(uint32_t (&a)[5], uint64_t b0, uint64_t b1)
{
    asm("add.cc.u32  %0, %0, %5;\n\t"
        "addc.cc.u32 %1, %1, %6;\n\t"
        "addc.cc.u32 %2, %2, %7;\n\t"
        "addc.cc.u32 %3, %3, %8;\n\t"
        "addc.u32    %4, %4, 0;"
        : "+r"(a[0]), "+r"(a[1]), "+r"(a[2]), "+r"(a[3]), "+r"(a[4])
        : "r"((uint32_t)b0), "r"((uint32_t)(b0 >> 32)), "r"((uint32_t)b1), "r"((uint32_t)(b1 >> 32)));
}

template <int NP>
__device__ __forceinline__ void crt_values(const uint32_t (&y)[NP], const CrtConst& K, uint64_t& c0,
                                           uint64_t& c1, uint64_t& c2)
{
    if constexpr (NP == 5 || NP == 6) {
        // X = sum_j y_j (P/p_j) - k P modulo 2^(32 NP), as 64-bit products of
        // 32-bit words summed without carries: y_j c < p_j 2^32, and the pairs
        // (0, 1), (2, 3) and (4, 5) of primes sum to less than 2^32 each, with
        // room for k (2^(32 NP) - P), k < 8, beside the last.  (One 64-bit
        // product-sum holds the FMA pipe for 4.3 cycles a warp where the low and
        // high halves by themselves take 6.)
        // k = round(sum_j y_j / p_j) from the top 23 bits of each y_j under the
        // exponent of 2^23: no integer-to-float conversions; off by less than
        // 10^-5, and the coefficient bound leaves 3 10^-4.
        float fk = K.koff;
#pragma unroll
        for (int jp = 0; jp < NP; jp++)
            fk = fmaf(__uint_as_float(__byte_perm(y[jp], 0x4bu, 0x4321)), K.kc[jp], fk);
        const uint32_t k = __float_as_uint(fk + 12582912.0f) & 0xffu;   // 1.5 2^23: rounds to an integer
        constexpr int CW = NP - 1;
        uint64_t g[3][CW];
#pragma unroll
        for (int w = 0; w < CW; w++) {
            g[0][w] = (uint64_t)y[0] * K.cof[0][w] + (uint64_t)y[1] * K.cof[1][w];
            g[1][w] = (uint64_t)y[2] * K.cof[2][w] + (uint64_t)y[3] * K.cof[3][w];
            g[2][w] = (uint64_t)y[4] * K.cof[4][w] + (uint64_t)k * K.Pneg[w];
            if constexpr (NP == 6) g[2][w] += (uint64_t)y[5] * K.cof[5][w];
        }
        // even words e (0 .. 3, carries into word 4), odd words o (1 .. 4, and
        // 5 for six primes)
        uint32_t e[5] = {(uint32_t)g[0][0], (uint32_t)(g[0][0] >> 32), (uint32_t)g[0][2], (uint32_t)(g[0][2] >> 32), 0};
        uint32_t o[5] = {(uint32_t)g[0][1], (uint32_t)(g[0][1] >> 32), (uint32_t)g[0][3], (uint32_t)(g[0][3] >> 32), 0};
#pragma unroll
        for (int t = 1; t < 3; t++) {
            add128c(e, g[t][0], g[t][2]);
            add128c(o, g[t][1], g[t][3]);
        }
        if constexpr (NP == 5) {
            e[4] += k * K.Pneg[4];
            asm("add.cc.u32  %0, %0, %4;\n\t"
                "addc.cc.u32 %1, %1, %5;\n\t"
                "addc.cc.u32 %2, %2, %6;\n\t"
                "addc.u32    %3, %3, %7;"
                : "+r"(e[1]), "+r"(e[2]), "+r"(e[3]), "+r"(e[4])
                : "r"(o[0]), "r"(o[1]), "r"(o[2]), "r"(o[3]));
            c2 = (uint64_t)e[4];
        } else {
            // words 4, 5: the products at word 4, the carries out of the even and
            // odd words below, and k Pneg at word 5
            const uint64_t top = g[0][4] + g[1][4] + g[2][4] + e[4] + ((uint64_t)(k * K.Pneg[5]) << 32) +
                                 ((uint64_t)o[4] << 32);
            uint32_t t4 = (uint32_t)top, t5 = (uint32_t)(top >> 32);
            asm("add.cc.u32  %0, %0, %5;\n\t"
                "addc.cc.u32 %1, %1, %6;\n\t"
                "addc.cc.u32 %2, %2, %7;\n\t"
                "addc.cc.u32 %3, %3, %8;\n\t"
                "addc.u32    %4, %4, 0;"
                : "+r"(e[1]), "+r"(e[2]), "+r"(e[3]), "+r"(t4), "+r"(t5)
                : "r"(o[0]), "r"(o[1]), "r"(o[2]), "r"(o[3]));
            c2 = (uint64_t)t4 | ((uint64_t)t5 << 32);
        }
        c0 = (uint64_t)e[0] | ((uint64_t)e[1] << 32);
        c1 = (uint64_t)e[2] | ((uint64_t)e[3] << 32);
        return;
    }
    float fk = 0.0f;
#pragma unroll
    for (int jp = 0; jp < NP; jp++) {
        fk = fmaf((float)y[jp], K.finv[jp], fk);
    }
    // P/p_j has NP-1 words (one when NP == 1); the sum has NP words.
    constexpr int CW = NP > 1 ? NP - 1 : 1;
    uint64_t acc[NP + 1];
#pragma unroll
    for (int w = 0; w <= NP; w++) acc[w] = 0;
#pragma unroll
    for (int jp = 0; jp < NP; jp++) {
#pragma unroll
        for (int w = 0; w < CW; w++) {
            const uint64_t pr = (uint64_t)y[jp] * K.cof[jp][w];
            acc[w] += (uint32_t)pr;
            acc[w + 1] += pr >> 32;
        }
    }
    const uint32_t k = (uint32_t)rintf(fk);
    uint32_t X[NP];
    uint64_t carry = 0;
#pragma unroll
    for (int w = 0; w < NP; w++) {
        const uint64_t t = acc[w] + carry;
        X[w] = (uint32_t)t;
        carry = t >> 32;
    }
    int64_t borrow = 0;
#pragma unroll
    for (int w = 0; w < NP; w++) {
        const int64_t t = (int64_t)X[w] - (int64_t)((uint64_t)k * K.P[w]) - borrow;
        X[w] = (uint32_t)t;
        borrow = -(t >> 32);
    }
    uint32_t W[6] = {0, 0, 0, 0, 0, 0};
#pragma unroll
    for (int w = 0; w < NP && w < 6; w++) W[w] = X[w];
    c0 = (uint64_t)W[0] | ((uint64_t)W[1] << 32);
    c1 = (uint64_t)W[2] | ((uint64_t)W[3] << 32);
    c2 = (uint64_t)W[4] | ((uint64_t)W[5] << 32);
}

// Look-back status word: [31:4] epoch, [3:2] state (1 aggregate, 2 inclusive),
// [1] generate / carry-out, [0] propagate.
constexpr uint32_t ST_AGG = 1u << 2, ST_INC = 2u << 2;
constexpr long LOOKBACK_SPIN_LIMIT = 1L << 22;
// Residue CRT/carry tiles: CRT_THREADS threads of 4 coefficients.  Measured
// on the B200 (2^24 x 2^24 product): 128-thread tiles 0.330 ms, 256 0.337,
// 512 0.377 -- smaller tiles keep more of them resident per SM while one
// waits on its ticket or look-back.  The recombination is what bounds them: with
// 64-bit product-sums (crt_values) 0.330 -> 0.289 ms, against 0.144 ms of HBM
// traffic; persistent CTAs that draw the next ticket and load its residues ahead
// were slower (0.349 ms: 72 registers and fewer CTAs per SM).
constexpr int CRT_THREADS = 128;
constexpr int CRT_TILE = 4 * CRT_THREADS;

// NP == 0 is the direct mode: the coefficient values are precomputed (the
// basecase kernel's column sums) instead of recombined from residues.
template <int NP, int THREADS>
__global__ void __launch_bounds__(THREADS)
k_crt_carry(const uint32_t* __restrict__ res, int logM, uint64_t L, uint64_t zn,
            uint64_t* __restrict__ z, CrtConst K, uint32_t* __restrict__ status,
            unsigned long long* __restrict__ ticket, unsigned long long ticket_base,
            uint32_t epoch, int* __restrict__ err,
            const InstDesc* __restrict__ desc, const uint32_t* __restrict__ tile_inst,
            uint64_t base)
{
    constexpr int PER = 4;
    constexpr int TILE = PER * THREADS;
    constexpr int NW = THREADS / 32;
    // last three coefficients of each warp (slot w + 1; slot 0 = the tile's
    // halo, coefficients n0 - 3 .. n0 - 1): c0, c1, c2 of the last, c1, c2 of
    // the one before, c2 of the one before that
    __shared__ uint64_t wlast[NW + 1][6];
    __shared__ uint32_t sh_tile;
    __shared__ uint32_t wg[NW], wp[NW];
    __shared__ uint32_t sh_carry_in;

    pdl_wait();
    if (threadIdx.x == 0) sh_tile = (uint32_t)(atomicAdd(ticket, 1ull) - ticket_base);
    __syncthreads();
    // `gtile` numbers tiles across the launch (status words, look-back order);
    // `tile` is the tile inside its product: a batch launch runs the tiles of
    // all its products back to back, and each product's first tile starts a
    // fresh carry chain, so look-backs never cross into the previous product.
    const uint32_t gtile = sh_tile;
    uint32_t tile = gtile;
    if (desc) {
        const InstDesc& D = desc[tile_inst[gtile]];
        tile = gtile - D.tile0;
        res = D.ra;
        L = D.an + D.bn - 1;
        zn = D.an + D.bn;
        z = D.z;
    }
    // coefficient / limb index of the tile's first position: a window product
    // starts at limb `base` (z[0] is limb base; limbs below it are not
    // produced and their carry into the window is not added -- the lower
    // approximation of a windowed product)
    const int64_t n0 = (int64_t)base + (int64_t)tile * TILE;
    // limbs below zn need coefficients below zn only; a window's transform
    // length covers min(L, zn) coefficients, not necessarily L
    L = L < zn ? L : zn;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;

    // this thread's coefficients n0 + 4t .. n0 + 4t + 3, kept in registers;
    // a thread's four residues per prime are one 16-byte load when they lie
    // inside the array
    uint64_t c0[PER], c1[PER], c2[PER];
    {
        const uint64_t nb = (uint64_t)(n0 + threadIdx.x * PER);
        if constexpr (NP == 0) {
            // direct mode: values given as three planes of 2^logM 64-bit words
#pragma unroll
            for (int q = 0; q < PER; q++) {
                c0[q] = c1[q] = c2[q] = 0;
                if (nb + q < L) crt_coeff<0>(res, logM, nb + q, K, c0[q], c1[q], c2[q]);
            }
        } else {
            uint32_t y[PER][NP];
            // 16-byte loads need nb % 4 == 0 (always true for whole products; a
            // window may start at any limb) and the four residues inside the array
            if ((nb & 3) == 0 && nb + PER <= ((uint64_t)1 << logM)) {
#pragma unroll
                for (int jp = 0; jp < NP; jp++) {
                    const uint4 v = *reinterpret_cast<const uint4*>(res + ((size_t)jp << logM) + nb);
                    y[0][jp] = v.x; y[1][jp] = v.y; y[2][jp] = v.z; y[3][jp] = v.w;
                }
            } else {
#pragma unroll
                for (int q = 0; q < PER; q++)
#pragma unroll
                    for (int jp = 0; jp < NP; jp++)
                        y[q][jp] = (nb + q < L) ? res[((size_t)jp << logM) + nb + q] : 0u;
            }
#pragma unroll
            for (int q = 0; q < PER; q++) {
                c0[q] = c1[q] = c2[q] = 0;
                if (nb + q < L) crt_values<NP>(y[q], K, c0[q], c1[q], c2[q]);
            }
        }
    }
    if (lane == 31) {
        uint64_t* w = wlast[warp + 1];
        w[0] = c0[3]; w[1] = c1[3]; w[2] = c2[3]; w[3] = c1[2]; w[4] = c2[2]; w[5] = c2[1];
    }
    if (threadIdx.x < 3) {
        // halo: coefficients n0 - 1, n0 - 2, n0 - 3 (zero before the product),
        // one per lane of warp 0 so the three CRTs run side by side
        const int d = threadIdx.x + 1;
        const int64_t n = n0 - d;
        uint64_t h0 = 0, h1 = 0, h2 = 0;
        if (n >= 0 && (uint64_t)n < L) crt_coeff<NP>(res, logM, (uint64_t)n, K, h0, h1, h2);
        uint64_t* w = wlast[0];
        if (d == 1) { w[0] = h0; w[1] = h1; w[2] = h2; }
        else if (d == 2) { w[3] = h1; w[4] = h2; }
        else { w[5] = h2; }
    }
    __syncthreads();
    // the previous thread's last three coefficients (shuffle, or the slot of
    // the previous warp / the halo for lane 0)
    uint64_t p0 = __shfl_up_sync(0xffffffffu, c0[3], 1);
    uint64_t p1 = __shfl_up_sync(0xffffffffu, c1[3], 1);
    uint64_t p2 = __shfl_up_sync(0xffffffffu, c2[3], 1);
    uint64_t q1 = __shfl_up_sync(0xffffffffu, c1[2], 1);
    uint64_t q2 = __shfl_up_sync(0xffffffffu, c2[2], 1);
    uint64_t r2 = __shfl_up_sync(0xffffffffu, c2[1], 1);
    if (lane == 0) {
        const uint64_t* w = wlast[warp];
        p0 = w[0]; p1 = w[1]; p2 = w[2]; q1 = w[3]; q2 = w[4]; r2 = w[5];
    }

    // limb n receives s_n = X0[n] + X1[n-1] + X2[n-2] = lo_n + 2^64 cr_n (cr_n <= 2),
    // and then t_n = lo_n + cr_(n-1): a single-bit carry chain remains.
    auto s3 = [](uint64_t a, uint64_t b, uint64_t c, uint64_t& lo) -> uint32_t {
        uint64_t s = a;
        uint32_t cr = 0;
        uint64_t t = s + b; cr += t < s; s = t;
        t = s + c; cr += t < s; s = t;
        lo = s;
        return cr;
    };
    // X0, X1, X2 of coefficients 4t - 3 .. 4t + 3 relative to the thread
    const uint64_t x0[5] = {p0, c0[0], c0[1], c0[2], c0[3]};               // coefficients 4t-1 .. 4t+3
    const uint64_t x1[6] = {q1, p1, c1[0], c1[1], c1[2], c1[3]};           // 4t-2 .. 4t+3
    const uint64_t x2[7] = {r2, q2, p2, c2[0], c2[1], c2[2], c2[3]};       // 4t-3 .. 4t+3
    uint64_t tv[PER];
    uint32_t gbits = 0, pbits = 0;
    {
        uint64_t lo_prev;
        // s at limb 4t - 1: X0[4t-1] + X1[4t-2] + X2[4t-3]
        uint32_t cr_prev = (n0 + threadIdx.x * PER >= 1) ? s3(x0[0], x1[0], x2[0], lo_prev) : 0;
#pragma unroll
        for (int q = 0; q < PER; q++) {
            uint64_t lo;
            const uint32_t cr = s3(x0[q + 1], x1[q + 1], x2[q + 1], lo);
            const uint64_t t = lo + cr_prev;
            const uint32_t g = t < lo;
            tv[q] = t;
            gbits |= g << q;
            pbits |= (uint32_t)(t == ~0ull) << q;
            cr_prev = cr;
        }
    }
    // thread aggregate (G, P) over its PER limbs, low to high
    uint32_t Gt = 0, Pt = 1;
    for (int q = 0; q < PER; q++) {
        const uint32_t g = (gbits >> q) & 1, pq = (pbits >> q) & 1;
        Gt = g | (pq & Gt);
        Pt = Pt & pq;
    }
    // inclusive warp scan of (G, P)
    uint32_t Gi = Gt, Pi = Pt;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
        const uint32_t Go = __shfl_up_sync(0xffffffffu, Gi, d);
        const uint32_t Po = __shfl_up_sync(0xffffffffu, Pi, d);
        if (lane >= d) { Gi = Gi | (Pi & Go); Pi = Pi & Po; }
    }
    if (lane == 31) { wg[warp] = Gi; wp[warp] = Pi; }
    __syncthreads();
    // exclusive prefix over warps (small, done redundantly per thread)
    uint32_t Gw = 0, Pw = 1;
    for (int w = 0; w < warp; w++) { Gw = wg[w] | (wp[w] & Gw); Pw = Pw & wp[w]; }
    // exclusive prefix for this thread within the tile
    uint32_t Ge = __shfl_up_sync(0xffffffffu, Gi, 1), Pe = __shfl_up_sync(0xffffffffu, Pi, 1);
    if (lane == 0) { Ge = 0; Pe = 1; }
    Ge = Ge | (Pe & Gw);
    Pe = Pe & Pw;

    if (threadIdx.x == THREADS - 1) {
        // tile aggregate = inclusive prefix of the last thread
        const uint32_t Gtile = Gi | (Pi & Gw);
        const uint32_t Ptile = Pi & Pw;
        uint32_t cin = 0;
        if (tile == 0) {
            __threadfence();
            atomicExch(&status[gtile], (epoch << 4) | ST_INC | (Gtile << 1));
        } else {
            atomicExch(&status[gtile], (epoch << 4) | ST_AGG | (Gtile << 1) | Ptile);
            uint32_t Gr = 0, Pr = 1;
            int64_t k = (int64_t)gtile - 1;
            long spins = 0;
            while (true) {
                const uint32_t st = *(volatile uint32_t*)&status[k];
                if ((st >> 4) != epoch || (st & (3u << 2)) == 0) {
                    if (++spins > LOOKBACK_SPIN_LIMIT) { atomicOr(err, DEV_ERR_CARRY); cin = 0; break; }
                    __nanosleep(64);
                    continue;
                }
                const uint32_t bg = (st >> 1) & 1, bp = st & 1;
                if ((st & (3u << 2)) == ST_INC) { cin = Gr | (Pr & bg); break; }
                Gr = Gr | (Pr & bg);
                Pr = Pr & bp;
                if (!Pr) { cin = Gr; break; }
                --k;
                if (k < 0) { cin = Gr; break; }
            }
            const uint32_t cout = Gtile | (Ptile & cin);
            atomicExch(&status[gtile], (epoch << 4) | ST_INC | (cout << 1));
        }
        sh_carry_in = cin;
    }
    __syncthreads();
    pdl_trigger();
    uint32_t c = Ge | (Pe & sh_carry_in);
    uint64_t v[PER];
#pragma unroll
    for (int q = 0; q < PER; q++) {
        v[q] = tv[q] + c;
        c = ((gbits >> q) & 1) | (((pbits >> q) & 1) & c);
    }
    const uint64_t nb = (uint64_t)(n0 + threadIdx.x * PER);
    uint64_t* dst = z + (nb - base);
    if (nb + PER <= zn && ((uintptr_t)dst & 15) == 0) {
        reinterpret_cast<ulonglong2*>(dst)[0] = make_ulonglong2(v[0], v[1]);
        reinterpret_cast<ulonglong2*>(dst)[1] = make_ulonglong2(v[2], v[3]);
    } else {
#pragma unroll
        for (int q = 0; q < PER; q++)
            if (nb + q < zn) dst[q] = v[q];
    }
}

// ---------------------------------------------------------------------------
// Calibration: the transforms' Gentleman-Sande butterfly (same form and pipe
// mix as the row passes) in a register-only loop, 16 values per thread, four
// levels per iteration -- the integer-pipe peak the product kernels are
// measured against.  Every value is stored at the end (out holds gridDim.x *
// blockDim.x * 16 words).
constexpr int CAL_ITERS = 256;

__global__ void __launch_bounds__(256)
k_bfly_rate(uint32_t* __restrict__ out, const uint2* __restrict__ tw, uint32_t p, uint32_t seed)
{
    constexpr int NV = 16;
    uint32_t x[NV];
    const uint32_t t = blockIdx.x * blockDim.x + threadIdx.x;
#pragma unroll
    for (int i = 0; i < NV; i++) x[i] = (seed * (t + 1) * (uint32_t)(2 * i + 7)) % p;
    uint32_t w[4], wq[4];
#pragma unroll
    for (int l = 0; l < 4; l++) { w[l] = tw[1 + l].x; wq[l] = tw[1 + l].y; }
    for (int it = 0; it < CAL_ITERS; it++) {
#pragma unroll
        for (int l = 0; l < 4; l++) {
            const int h = 1 << l;
#pragma unroll
            for (int i = 0; i < NV; i++)
                if (!(i & h)) bfly_gs<ROW_GS_FMA_ADDS>(x[i], x[i + h], w[l], wq[l], p);
        }
    }
    uint32_t* o = out + (size_t)t * NV;
#pragma unroll
    for (int i = 0; i < NV; i++) o[i] = x[i];
}

}  // namespace fb
