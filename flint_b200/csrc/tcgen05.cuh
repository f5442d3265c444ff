// Byte-matrix products on the tensor cores (tcgen05, kind::i8) for transforms
// modulo 31-bit primes.
//
// A length-32 transform is the product of a fixed 32 x 32 matrix with every
// group of 32 residues.  A residue in memory is four unsigned bytes, so 32 of
// them are one 128-byte row of the A operand as they lie, whatever 32-bit
// representative they hold.  The B operand W holds byte c of
// w^(j k) 2^(8 b) mod p at row 4 k + c, column 4 j + b; the product's columns
// 4 k .. 4 k + 3 are then four sums S_c < 128 255^2 < 2^23 with
//     S_0 + 2^8 S_1 + 2^16 S_2 + 2^24 S_3 = sum_j x_j w^(j k)  (mod p),
// exact in 32-bit integers.  tc_reduce brings that 48-bit value below 2 p.
//
// Instruction and descriptor forms follow the PTX ISA's tcgen05 chapter:
// M = 128 rows from shared memory (128-byte rows, 128-byte swizzle), N = 128,
// K = 32 bytes per instruction, accumulators in TMEM.
#pragma once
#include <math.h>
#include <stdint.h>

namespace fb {

constexpr int TC_ROW_BYTES = 128;             // one A or W row: 32 residues
constexpr int TC_W_BYTES = 128 * TC_ROW_BYTES;
constexpr int TC_TILE_BYTES = 128 * TC_ROW_BYTES;   // 128 rows of A

__device__ __forceinline__ uint32_t tc_smem(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

// word offset of word `pos` of a buffer of 32-word rows under the 128-byte
// swizzle: 16-byte chunk q of row r sits at chunk q ^ (r & 7)
__device__ __forceinline__ constexpr int tc_swz(int pos) { return pos ^ (((pos >> 5) & 7) << 2); }

__device__ __forceinline__ void tc_mbar_init(uint32_t bar)
{
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(bar) : "memory");
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}

// Waits for the barrier's phase; false after a bounded number of polls (each
// suspends for a while in hardware, so the bound is far beyond any matrix
// product's time).
__device__ __forceinline__ bool tc_mbar_wait(uint32_t bar, uint32_t parity)
{
    for (int it = 0; it < (1 << 20); it++) {
        uint32_t ok;
        asm volatile("{\n\t.reg .pred p;\n\t"
                     "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
                     "selp.u32 %0, 1, 0, p;\n\t}"
                     : "=r"(ok)
                     : "r"(bar), "r"(parity)
                     : "memory");
        if (ok) return true;
    }
    return false;
}

// shared-memory writes of this thread become visible to the tensor core's reads
__device__ __forceinline__ void tc_fence_smem() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }

// TMEM columns (a power of two, at least 32), by one whole warp
__device__ __forceinline__ void tc_alloc(uint32_t smem_dst, uint32_t ncols)
{
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_dst), "r"(ncols)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tc_dealloc(uint32_t taddr, uint32_t ncols)
{
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(ncols) : "memory");
}

// the barrier completes its phase once every product issued so far is done
__device__ __forceinline__ void tc_commit(uint32_t bar)
{
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar) : "memory");
}

// K-major operand rows of 128 bytes, 128-byte swizzle: atoms of 8 rows (1024
// bytes, the stride field), base a multiple of 1024 bytes
__device__ __forceinline__ uint64_t tc_desc(uint32_t addr)
{
    return (uint64_t)((addr & 0x3ffffu) >> 4) | (1ull << 16) | (64ull << 32) | (1ull << 46) | (2ull << 61);
}

// D[128 x 128] = A[128 x 128 bytes] W^T, unsigned bytes into 32-bit sums; one thread
__device__ __forceinline__ void tc_mma_tile(uint32_t d, uint32_t a_smem, uint32_t w_smem)
{
    // 32-bit integer accumulators, unsigned operands, N = 128, M = 128
    constexpr uint32_t idesc = (2u << 4) | ((128u >> 3) << 17) | ((128u >> 4) << 24);
    const uint64_t a = tc_desc(a_smem), w = tc_desc(w_smem);
#pragma unroll
    for (int k = 0; k < 4; k++)   // 32 bytes of K per instruction
        asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.u32 p, %4, 0;\n\t"
                     "tcgen05.mma.cta_group::1.kind::i8 [%0], %1, %2, %3, p;\n\t}" ::"r"(d),
                     "l"(a + 2 * k), "l"(w + 2 * k), "r"(idesc), "r"(k)
                     : "memory");
}

// 32 columns of this warp's 32 TMEM lanes: thread l gets lane l's words.  The
// load is asynchronous: its wait stands in the same statement, so that nothing
// that uses r can be scheduled between the two.
__device__ __forceinline__ void tc_ld32(uint32_t (&r)[32], uint32_t taddr)
{
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
        "{%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,"
        "%28,%29,%30,%31}, [%32];\n\t"
        "tcgen05.wait::ld.sync.aligned;"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
          "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]),
          "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]),
          "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
        : "r"(taddr)
        : "memory");
}

// Quotient constants of a prime: c = 2^24 / p, m = 2^23 + 1 - 2^23 c - 1/2 - e
// with e in [0.02, 0.53] (m is a multiple of 1/2), kp = 0x4b000001 p mod 2^32.
struct TcPrime {
    float c, m;
    uint32_t kp;
};

// v = S_0 + 2^8 S_1 + 2^16 S_2 + 2^24 S_3 (S < 2^23) modulo p, in [0, 1.6 p).
// q = round(t c - 1/2 - e) >= -1, t = floor(v 2^-24) < 2^23: with t's bits under
// the exponent of 2^23 the fused multiply-add returns 2^23 + 1 + q exactly
// rounded (at least 2^23, where floats step by 1), and v / p - q lies in
// [e - 0.01, 1 + e + 0.03].  The quotient stays in its float bits
// (0x4b000001 + q); kp takes the bias out.
__device__ __forceinline__ uint32_t tc_reduce(uint32_t s0, uint32_t s1, uint32_t s2, uint32_t s3, uint32_t p,
                                              const TcPrime& K)
{
    const uint32_t lo = s0 + (s1 << 8), hi = s2 + (s3 << 8);        // both below 2^31
    const uint32_t w = hi + (lo >> 16);                             // floor(v 2^-16) < 2^31
    const float t = __uint_as_float(__byte_perm(w, 0x4bu, 0x4321));  // 2^23 + (w >> 8)
    const uint32_t q = __float_as_uint(__fmaf_rn(t, K.c, K.m));
    return (K.kp - q * p) + (lo + (hi << 16));
}

// host: the constants of a prime
static inline TcPrime tc_prime(uint32_t p)
{
    TcPrime K;
    K.c = 16777216.0f / (float)p;
    K.m = (float)(floor((8388608.0 * (1.0 - (double)K.c) + 0.5 - 0.02) * 2.0) * 0.5);
    K.kp = 0x4b000001u * p;
    return K;
}

// host: the W of a prime for the row and column kernels' five lowest levels
// (natural order in, bit-reversed out: output m has frequency bitrev5(m)),
// as its swizzled shared-memory image; w32 has order 32.
static inline void tc_fill_w(uint8_t* img, uint32_t w32, uint32_t p)
{
    uint32_t pw[32];
    pw[0] = 1;
    for (int k = 1; k < 32; k++) pw[k] = (uint32_t)((uint64_t)pw[k - 1] * w32 % p);
    for (int m = 0; m < 32; m++) {
        int f = 0;
        for (int b = 0; b < 5; b++) f |= ((m >> b) & 1) << (4 - b);
        for (int j = 0; j < 32; j++)
            for (int b = 0; b < 4; b++) {
                const uint32_t v = (uint32_t)(((uint64_t)pw[(j * f) & 31] << (8 * b)) % p);
                for (int c = 0; c < 4; c++) {
                    const int n = 4 * m + c, kb = 4 * j + b;
                    img[n * TC_ROW_BYTES + (((kb >> 4) ^ (n & 7)) << 4) + (kb & 15)] = (uint8_t)(v >> (8 * c));
                }
            }
    }
}

}  // namespace fb
