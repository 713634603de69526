// pg_tc.cuh -- strong base-2 tests of candidates n = m*K + X with the
// reduction on the tensor cores.
//
// A Montgomery squaring of an L-word number spends two thirds of its word
// products on the reduction, against a modulus that differs from lane to
// lane.  Here every candidate of a window shares K, and only the small m and
// X differ, so the reduction becomes two products with fixed numbers, each a
// matrix product of the CTA's 128 values (rows of bytes) with the Toeplitz
// matrix of the fixed number's bytes: u8 x u8 -> s32 on tcgen05, exact.
//
// One step takes y < 2.22 n to r = 2^b * (m*T - z*n), T = y^2:
//   T   = y^2                                  L(L+1)/2 word products (integer pipe)
//   q   = T_hi * mu / 2^..                     matrix 1: mu = floor(2^u / K), T_hi = T >> 32 (L-4)
//   z   = floor(q - X*q/n - 1/16)              double precision on the top words of q
//   w   = T - z*K  (mod 2^32L)                 matrix 2: K
//   r   = 2^b * (m*w - X*z)  (mod 2^32L)       2L word products
// q falls short of T/K by at most 2^-8 + 2^-16 (the cut ends of T and mu, and
// the columns left out below its guard word), T/K - X*T/(K*n) = m*T/n, and
// the correction's own rounding is below 2^-5 (pick_tc in pg_dispatch.cu
// states the sizes), so m*T/n - z lies in [1/32, 1.11) and
// r / 2^b = m*T - z*n = m*(T - z*K) - z*X in [0, 1.11 n): its low L words hold
// it, and the next y is below 2.22 n.  r is m*T mod n: with y standing for
// x*m^-1 mod n the step maps x to 2^b * x^2, so a test starts from
// 2^e * m^-1 mod n = s*K + (s*X + 2^e)/m, s = -2^e * X^-1 mod m, for the leading
// bits e of the exponent, and compares with +-m^-1 (e = 0) at the end.
#pragma once

#include "pg_internal.h"
#include "pg_mont.cuh"

namespace pg {

constexpr double TC_MARGIN = 1.0 / 16;
constexpr int TC_ROWS = 128;  // numbers per CTA: one thread, one TMEM lane, one matrix row each

template <int L>
struct TcDim {
    static constexpr int HW = L - 4;                         // T_hi = T >> 32*HW
    static constexpr int TOP = 5;                            // words of z the correction reads
    static constexpr int NT = 2 * L - HW;                    // words of T_hi
    static constexpr int NZ = L + 1;                         // words of z
    static constexpr int K1 = (4 * NT + 31) / 32 * 32;       // bytes per row of matrix 1's input
    static constexpr int N1 = (4 + 4 * NZ + 15) / 16 * 16;   // its output columns: a guard word, then z's words
    static constexpr int K2 = (4 * NZ + 31) / 32 * 32;
    static constexpr int N2 = (4 * L + 15) / 16 * 16;
    static constexpr int NMAX = N1 > N2 ? N1 : N2;
    static constexpr int COLS = NMAX <= 32 ? 32 : NMAX <= 64 ? 64 : NMAX <= 128 ? 128 : 256;  // TMEM columns
    // a column of D sums at most 4 NT products of two bytes; tc_words needs a
    // pair of columns with what moved up from the pair below in 32 bits (so up
    // to 256 bytes, L = 60; 192 at L = 44)
    static_assert(257ull * (4 * NT) * 255 * 255 + 65535 <= 0xffffffffull, "columns too large for tc_words");
    static constexpr int A_BYTES = TC_ROWS * (K1 > K2 ? K1 : K2);
    static constexpr int SMEM = A_BYTES + N1 * K1 + N2 * K2;
};

// ---------------------------------------------------------------- tcgen05

__device__ __forceinline__ uint32_t smem_u32(const void *p) { return (uint32_t)__cvta_generic_to_shared(p); }

// shared-memory matrix descriptor, K-major, no swizzle: 8 x 16 B core
// matrices, lbo bytes apart along K and 128 B apart along rows
__device__ __forceinline__ uint64_t tc_desc(uint32_t addr, uint32_t lbo) {
    return (uint64_t)((addr >> 4) & 0x3fffu) | ((uint64_t)(lbo >> 4) << 16) | ((uint64_t)(128u >> 4) << 32) |
           (1ull << 46);
}

// one instruction: D (s32, 128 x N) = or += A (u8, 128 x 32) * B^T (u8, N x 32)
template <int N>
__device__ __forceinline__ void tc_mma1(uint32_t d, uint64_t ad, uint64_t bd, uint32_t accumulate) {
    constexpr uint32_t idesc = (2u << 4) | ((uint32_t)(N / 8) << 17) | ((uint32_t)(TC_ROWS / 16) << 24);
    asm volatile(
        "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::i8 [%0], %1, %2, %3, p;\n\t}" ::"r"(d), "l"(ad), "l"(bd), "r"(idesc),
        "r"(accumulate));
}

// D = A * B^T for a Toeplitz matrix B (N rows of KB bytes), 32 bytes of A an
// instruction, leaving out the columns where that part of B is zero.  LOWER:
// B[c][k] is zero for c < k, so bytes 32k.. reach the columns from 32k on; the
// first instruction writes all columns.  Otherwise B[c][k] is zero for
// c > k, bytes 32k.. reach the columns below 32k + 32 and the last
// instruction comes first.  Against whole products: 0.67 of the tensor work at
// L = 23, 0.56 at L = 40; the integer pipes wait for about a tenth of a step
// while all of it runs (measured by issuing it twice).
template <int N, int KB, bool LOWER, int K = 0>
__device__ __forceinline__ void tc_mma(uint32_t d, uint32_t a, uint32_t b) {
    constexpr int STEPS = KB / 32, k = LOWER ? K : STEPS - 1 - K;
    if constexpr (K < STEPS && (!LOWER || 32 * k < N)) {
        constexpr int C0 = LOWER ? 32 * k : 0;
        constexpr int C1 = LOWER || K == 0 || 32 * k + 32 > N ? N : 32 * k + 32;
        tc_mma1<C1 - C0>(d + C0, tc_desc(a + k * 2 * TC_ROWS * 16, TC_ROWS * 16),
                         tc_desc(b + k * 2 * N * 16 + C0 * 16, N * 16), K);
        tc_mma<N, KB, LOWER, K + 1>(d, a, b);
    }
}
__device__ __forceinline__ void tc_commit(uint32_t mbar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(mbar) : "memory");
}
__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }

// Waits for the mbarrier's phase; false when it did not come within the limit.
__device__ __forceinline__ bool tc_wait(uint32_t mbar, uint32_t phase) {
    for (uint32_t i = 0; i < (1u << 18); i++) {
        uint32_t ok;
        asm volatile(
            "{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
            "selp.u32 %0, 1, 0, p;\n\t}" : "=r"(ok) : "r"(mbar), "r"(phase) : "memory");
        if (ok) return true;
    }
    return false;
}

// 16 columns of this thread's TMEM lane
__device__ __forceinline__ void tc_ld16(uint32_t (&v)[16], uint32_t addr) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
        : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]), "=r"(v[8]),
          "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15])
        : "r"(addr));
}
__device__ __forceinline__ void tc_wait_ld() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }

// ------------------------------------------------------------- arithmetic

// T = x^2 (2L words).  Cross products once in two arrays of aligned register
// pairs (as in mont_sqr), merged, doubled, then the diagonal in one chain.
template <int L>
__device__ __forceinline__ void tc_square(const uint32_t (&x)[L], uint32_t (&T)[2 * L]) {
    uint32_t E[2 * L + 2], F[2 * L + 2];
#pragma unroll
    for (int k = 0; k < 2 * L + 2; k++) E[k] = F[k] = 0;
#pragma unroll
    for (int i = 0; i < L - 1; i++) {
        const uint32_t a = x[i];
#pragma unroll
        for (int c = 0; c < 2; c++) {
            const int j0 = i + 1 + c;
            if (j0 >= L) continue;
            const int jl = j0 + ((L - 1 - j0) / 2) * 2;
            const bool top = jl == L - 1;
#pragma unroll
            for (int j = j0; j < L; j += 2) {
                const int p = i + j;
                uint32_t &lo = (p & 1) == 0 ? E[p] : F[p - 1];
                uint32_t &hi = (p & 1) == 0 ? E[p + 1] : F[p];
                lo = j == j0 ? mad_lo_cc(a, x[j], lo) : madc_lo_cc(a, x[j], lo);
                hi = (j == jl && top) ? madc_hi(a, x[j], hi) : madc_hi_cc(a, x[j], hi);
            }
            if (!top) {
                const int cp = i + jl + 2;
                if ((cp & 1) == 0)
                    E[cp] = addc(E[cp], 0u);
                else
                    F[cp - 1] = addc(F[cp - 1], 0u);
            }
        }
    }
    T[0] = E[0];
    T[1] = add_cc(E[1], F[0]);
#pragma unroll
    for (int k = 2; k < 2 * L; k++) T[k] = k + 1 < 2 * L ? addc_cc(E[k], F[k - 1]) : addc(E[k], F[k - 1]);
#pragma unroll
    for (int k = 2 * L - 1; k >= 1; k--) T[k] = __funnelshift_l(T[k - 1], T[k], 1);
    T[0] <<= 1;
    mad_link<true>(T[0], T[1], x[0], x[0]);
#pragma unroll
    for (int i = 1; i < L; i++) {
        T[2 * i] = madc_lo_cc(x[i], x[i], T[2 * i]);
        T[2 * i + 1] = i + 1 < L ? madc_hi_cc(x[i], x[i], T[2 * i + 1]) : madc_hi(x[i], x[i], T[2 * i + 1]);
    }
}

// NW words from the byte columns of the D matrix from column 0 on: four
// columns (each below 2^24, TcDim) make a word.  With p0 = c0 + c1*2^8 and
// p1 = c2 + c3*2^8 the value is the sum of two word strings, p0 plus the high
// half of the p1 below it (below 2^32, TcDim), and p1's low half moved up: one
// carry chain, so no 64-bit multiply (p1 * 2^16 + p0) adds to the multiply
// pipe's load: 2507 -> 2234 cycles a step at L = 23.  Columns are read 16 at a
// time, three reads in flight.
template <int NW>
__device__ __forceinline__ void tc_words(uint32_t (&out)[NW], uint32_t taddr) {
    constexpr int G = (4 * NW + 15) / 16;
    uint32_t carry = 0, up = 0;
#pragma unroll
    for (int g0 = 0; g0 < G; g0 += 3) {
        uint32_t v[3][16], u[12], t[12];
#pragma unroll
        for (int g = 0; g < 3; g++)
            if (g0 + g < G) tc_ld16(v[g], taddr + 16 * (g0 + g));
        tc_wait_ld();
#pragma unroll
        for (int k = 0; k < 12; k++) {
            if (4 * g0 + k >= NW) continue;
            const uint32_t *c = &v[k / 4][4 * (k % 4)];
            const uint32_t p1 = c[2] + (c[3] << 8);
            u[k] = c[0] + (c[1] << 8) + up;
            t[k] = p1 << 16;
            up = p1 >> 16;
        }
        if (g0) (void)add_cc(carry, 0xffffffffu);
#pragma unroll
        for (int k = 0; k < 12; k++) {
            if (4 * g0 + k >= NW) continue;
            out[4 * g0 + k] = g0 + k == 0 ? add_cc(u[k], t[k]) : addc_cc(u[k], t[k]);
        }
        if (g0 + 3 < G) carry = addc(0u, 0u);
    }
}

// this thread's row of the A matrix: NW words, 16 B chunks TC_ROWS*16 apart
template <int NW>
__device__ __forceinline__ void tc_put_row(uint32_t arow, const uint32_t *w) {
#pragma unroll
    for (int c = 0; c < (NW + 3) / 4; c++) {
        uint32_t v[4];
#pragma unroll
        for (int k = 0; k < 4; k++) v[k] = 4 * c + k < NW ? w[4 * c + k] : 0u;
        asm volatile("st.shared.v4.b32 [%0], {%1,%2,%3,%4};" ::"r"(arow + c * TC_ROWS * 16), "r"(v[0]), "r"(v[1]),
                     "r"(v[2]), "r"(v[3]) : "memory");
    }
}

// Toeplitz matrix of the bytes of f (nw words): B[c][k] = byte (off + c - k)
// of f, zero outside it and for k >= kuse, rows of KB bytes in 16 B chunks
// N*16 apart.
template <int N, int KB>
__device__ __forceinline__ void tc_toeplitz(uint8_t *b, const uint32_t *f, int nw, int off, int kuse) {
    for (int i = threadIdx.x; i < N * (KB / 16); i += blockDim.x) {
        const int c = i % N, ch = i / N;
        uint32_t v[4] = {0, 0, 0, 0};
        for (int t = 0; t < 16; t++) {
            const int k = ch * 16 + t, p = off + c - k;
            if (k < kuse && p >= 0 && p < 4 * nw) v[t >> 2] |= ((f[p >> 2] >> (8 * (p & 3))) & 255u) << (8 * (t & 3));
        }
        *reinterpret_cast<uint4 *>(b + (size_t)ch * N * 16 + c * 16) = make_uint4(v[0], v[1], v[2], v[3]);
    }
}

// The shared pieces of a CTA.
struct TcShared {
    uint64_t mbar;
    uint32_t tmem;
    int32_t win;      // the window the CTA takes items from, -1 = none left
    int32_t bmax[4];  // per warp: largest bit length among its candidates
};

struct TcState {
    uint32_t a, b1, b2, mbar, tmem, arow, phase;  // shared addresses, TMEM base, this thread's row, next parity
    uint32_t taddr;                               // this warp's lanes of the TMEM columns
    bool lead;                                    // the thread that issues the matrix instructions
    bool ok;
};

// One squaring of every row of the CTA (all 128 threads call it).  m < 2^30,
// xabs < 2^24; ratio = -X * 2^(32 (NZ-TOP)) / n.  A wait that ran out clears
// S.ok; the threads agree on it at the next barrier, and the call that holds
// that barrier returns false in all of them.
template <int L>
__device__ __forceinline__ bool tc_step(TcState &S, uint32_t (&y)[L], uint32_t m, uint32_t xabs, uint32_t xneg,
                                        double ratio, uint32_t dbl) {
    using D = TcDim<L>;
    uint32_t T[2 * L];
    tc_square<L>(y, T);
    tc_put_row<D::NT>(S.arow, T + D::HW);
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    tc_fence_before();
    S.ok = __syncthreads_and(S.ok);
    if (!S.ok) return false;
    if (S.lead) {
        tc_fence_after();
        tc_mma<D::N1, D::K1, false>(S.tmem, S.a, S.b1);
        tc_commit(S.mbar);
    }
    S.ok &= tc_wait(S.mbar, S.phase);
    S.phase ^= 1;
    tc_fence_after();
    uint32_t q[D::NZ + 1], z[D::NZ];  // the quotient T/K: a fraction word, then its integer part
    tc_words<D::NZ + 1>(q, S.taddr);
#pragma unroll
    for (int k = 0; k < D::NZ; k++) z[k] = q[k + 1];
    {  // z += floor(fraction - X*z/n - margin), from z's top words
        double top = (double)z[D::NZ - 1];
#pragma unroll
        for (int k = 2; k <= D::TOP; k++) top = __fma_rn(top, 4294967296.0, (double)z[D::NZ - k]);
        const double frac = __fma_rn((double)q[0], 0x1p-32, -TC_MARGIN);
        const long long t = __double2ll_rd(__fma_rn(ratio, top, frac));
        const uint32_t ext = (uint32_t)(t >> 63);
        z[0] = add_cc(z[0], (uint32_t)t);
        z[1] = addc_cc(z[1], (uint32_t)((unsigned long long)t >> 32));
#pragma unroll
        for (int k = 2; k < D::NZ; k++) z[k] = k + 1 < D::NZ ? addc_cc(z[k], ext) : addc(z[k], ext);
    }
    tc_put_row<D::NZ>(S.arow, z);
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    tc_fence_before();
    S.ok = __syncthreads_and(S.ok);
    if (!S.ok) return false;
    if (S.lead) {
        tc_fence_after();
        tc_mma<D::N2, D::K2, true>(S.tmem, S.a, S.b2);
        tc_commit(S.mbar);
    }
    // 2^b * (-X*z): products with |X|; z negated (two's complement) for X > 0
    const uint32_t mb = m << dbl, xb = xabs << dbl;
    uint64_t v[L];
#pragma unroll
    for (int k = 0; k < L; k++) v[k] = (uint64_t)xb * (z[k] ^ ~xneg);
    v[0] += xb & ~xneg;
    S.ok &= tc_wait(S.mbar, S.phase);
    S.phase ^= 1;
    tc_fence_after();
    uint32_t w[L];
    tc_words<L>(w, S.taddr);
    w[0] = sub_cc(T[0], w[0]);
#pragma unroll
    for (int k = 1; k < L; k++) w[k] = k + 1 < L ? subc_cc(T[k], w[k]) : subc(T[k], w[k]);
#pragma unroll
    for (int k = 0; k < L; k++) v[k] += (uint64_t)mb * w[k];
    y[0] = (uint32_t)v[0];
    y[1] = add_cc((uint32_t)v[1], (uint32_t)(v[0] >> 32));
#pragma unroll
    for (int k = 2; k < L; k++)
        y[k] = k + 1 < L ? addc_cc((uint32_t)v[k], (uint32_t)(v[k - 1] >> 32))
                         : addc((uint32_t)v[k], (uint32_t)(v[k - 1] >> 32));
    return true;
}

// j = -X^-1 mod m (X = +-xabs); false when gcd(m, X) > 1
__device__ __forceinline__ bool tc_inverse(uint32_t m, uint32_t xabs, bool neg, uint32_t &j) {
    uint32_t r0 = m, r1 = xabs % m;
    int64_t t0 = 0, t1 = 1;
    while (r1) {
        const uint32_t q = r0 / r1, r2 = r0 - q * r1;
        const int64_t t2 = t0 - (int64_t)q * t1;
        r0 = r1;
        r1 = r2;
        t0 = t1;
        t1 = t2;
    }
    if (r0 != 1) return false;
    // t0 * xabs = 1 mod m; -X^-1 = -t0 for X = xabs, t0 for X = -xabs
    int64_t v = neg ? t0 : -t0;
    v %= (int64_t)m;
    if (v < 0) v += m;
    j = (uint32_t)v;
    return true;
}

// y = s*K + (s*X + rho)/m (exact) + q, q in local memory or NULL
template <int L>
__device__ __forceinline__ void tc_start(uint32_t (&y)[L], const uint32_t *K, uint32_t s, uint32_t m, int64_t X,
                                         uint32_t rho, const uint32_t *q) {
    const int64_t c = ((int64_t)s * X + rho) / (int64_t)m;
    uint32_t carry = 0;
#pragma unroll
    for (int i = 0; i < L; i++) {
        uint64_t p = (uint64_t)__ldg(K + i) * s + carry;
        if (q) p += q[i];
        y[i] = (uint32_t)p;
        carry = (uint32_t)(p >> 32);
    }
    const uint32_t ext = (uint32_t)(c >> 63);
    y[0] = add_cc(y[0], (uint32_t)c);
    y[1] = addc_cc(y[1], (uint32_t)((uint64_t)c >> 32));
#pragma unroll
    for (int i = 2; i < L; i++) y[i] = i + 1 < L ? addc_cc(y[i], ext) : addc(y[i], ext);
}

// Helpers on words in local memory, rolled loops: a few calls per test.

// q = floor(2^e / m), e < 32L, m < 2^30; returns 2^e mod m
template <int L>
__device__ __noinline__ uint32_t tc_pow2_div(uint32_t *q, uint32_t e, uint32_t m) {
    const uint64_t inv = ~0ull / m;
    uint32_t rem = 0;
    for (int i = L - 1; i >= 0; i--) {
        uint32_t d = 0;
        if (i <= (int)(e >> 5)) {
            const uint64_t v = ((uint64_t)rem << 32) | (i == (int)(e >> 5) ? 1u << (e & 31) : 0u);
            uint64_t t = __umul64hi(v, inv), r = v - t * m;  // t falls short of v / m by less than 2
            while (r >= m) {
                t++;
                r -= m;
            }
            d = (uint32_t)t;
            rem = (uint32_t)r;
        }
        q[i] = d;
    }
    return rem;
}

// x < y
template <int L>
__device__ __forceinline__ bool tc_less(const uint32_t *x, const uint32_t *y) {
    for (int k = L - 1; k > 0; k--)
        if (x[k] != y[k]) return x[k] < y[k];
    return x[0] < y[0];
}

// x -= y; returns the borrow
template <int L>
__device__ __forceinline__ uint32_t tc_sub(uint32_t *x, const uint32_t *y) {
    uint32_t borrow = 0;
    for (int k = 0; k < L; k++) {
        const uint64_t d = (uint64_t)x[k] - y[k] - borrow;
        x[k] = (uint32_t)d;
        borrow = (uint32_t)(d >> 63);
    }
    return borrow;
}

// 1 when y = a mod n, 2 when y = -a mod n, else 0 (y < 8n is reduced in place; a < n)
template <int L>
__device__ __noinline__ int tc_compare(uint32_t *y, const uint32_t *a, const uint32_t *n) {
    for (int it = 0; it < 8 && !tc_less<L>(y, n); it++) tc_sub<L>(y, n);
    uint32_t d1 = 0, d2 = 0, carry = 0;
    for (int k = 0; k < L; k++) {
        d1 |= y[k] ^ a[k];
        const uint64_t t = (uint64_t)y[k] + a[k] + carry;
        d2 |= (uint32_t)t ^ n[k];
        carry = (uint32_t)(t >> 32);
    }
    return d1 == 0 ? 1 : (d2 | carry) == 0 ? 2 : 0;
}

}  // namespace pg
