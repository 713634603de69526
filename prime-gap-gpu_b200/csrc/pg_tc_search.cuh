// pg_tc_search.cuh -- the persistent search on tensor-core reductions
// (pg_tc.cuh): the work items, refill and first-prime rule of
// k_search_persistent (pg_search.cuh), with a CTA of 128 lanes instead of a
// warp holding 128 items of one window and testing them in step.
//
// Each L is instantiated in its own translation unit (pg_tcinst.cu with
// -DPG_TCL=L); pg_dispatch.cu maps a launch's operand size to one.
#pragma once

#include "pg_search.cuh"
#include "pg_tc.cuh"

namespace pg {

// CTAs per SM ptxas allots registers for
constexpr int tc_min_blocks(int L) { return L <= 24 ? 4 : L <= 28 ? 3 : 2; }

// The window whose queue is furthest behind (in candidates per side) among
// those with items left, the current one where it is within one candidate of
// that; -1 when every queue has run out.  Called by one warp.
__device__ __forceinline__ int tc_pick_window(const SearchArgs &a, uint32_t kspan, int cur) {
    const uint32_t lane = threadIdx.x & 31;
    uint32_t best = 0xffffffffu, cur_k = 0xffffffffu;
    int best_w = -1;
    for (uint32_t w = lane; w < a.n_win; w += 32) {
        const uint32_t n = a.win[w].nsides;
        const unsigned long long head = *(volatile const unsigned long long *)&a.win_next[w];
        if (n == 0 || head >= (unsigned long long)n * kspan) continue;
        const uint32_t k = (uint32_t)(head / n);
        if (k < best) {
            best = k;
            best_w = (int)w;
        }
        if ((int)w == cur) cur_k = k;
    }
    cur_k = __reduce_min_sync(0xffffffffu, cur_k);
    const uint32_t lo = __reduce_min_sync(0xffffffffu, best);
    if (lo == 0xffffffffu) return -1;
    if (cur_k != 0xffffffffu && cur_k <= lo + 1) return cur;
    const unsigned at = __ballot_sync(0xffffffffu, best == lo);
    return __shfl_sync(0xffffffffu, best_w, __ffs(at) - 1);
}

// What bounds it: the integer multiply pipe (L(L+1)/2 + 2L word products a
// step, over whole searches 53 % busy with two CTAs of L = 22 on an SM, 68 % with
// three of L = 23 and 70 % with two of L = 40) together with the register ports
// that the carry chains and column sums load beside it; the tensor pipe is 7 to
// 10 % busy and DRAM idle.  In a loop of steps alone one takes 2 228 SM-quarter
// cycles per warp at L = 23 with four CTAs on an SM (1 877 with the matrix round
// trips left out), at L = 40 5 513 with two; a Montgomery squaring with the
// reduction on the multiply pipe takes 3 600 and 12 400.  A step alone
// takes 3 800 cycles (two matrix round trips, the carry chains), so as many
// CTAs as TMEM and registers hold share an SM.  Searches of P = 257 .. 947
// (12 .. 44 words) run 1.2 .. 2.2 times as fast as on the one-warp kernel,
// which keeps the draining launches and the sizes pick_tc refuses.
template <int L>
__global__ void __launch_bounds__(TC_ROWS, tc_min_blocks(L)) k_search_tc(const __grid_constant__ SearchArgs a) {
    using D = TcDim<L>;
    extern __shared__ __align__(128) uint8_t sm[];
    __shared__ TcShared sh;
    const unsigned FULL = 0xffffffffu;
    const int tid = threadIdx.x;
    const uint32_t lane = tid & 31;
    uint8_t *const b1 = sm + D::A_BYTES, *const b2 = b1 + D::N1 * D::K1;
    if (tid < 32) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&sh.tmem)),
                     "r"((uint32_t)D::COLS) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
    }
    if (tid == 0) {
        asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_u32(&sh.mbar)) : "memory");
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    TcState S;
    S.a = smem_u32(sm);
    S.b1 = smem_u32(b1);
    S.b2 = smem_u32(b2);
    S.mbar = smem_u32(&sh.mbar);
    S.tmem = sh.tmem;
    S.arow = S.a + tid * 16;
    S.phase = 0;
    S.taddr = sh.tmem + ((uint32_t)(tid & ~31) << 16);
    S.lead = tid == 0;
    S.ok = true;

    uint32_t kspan = a.kspan;
    if (a.max_count) kspan = min(kspan, *a.max_count + a.ext_max);
    unsigned long long ntests = 0;
    int cur = -1;
    while (true) {
        if (tid < 32) {
            bool stop = false;
            int w = tc_pick_window(a, kspan, cur);
            if (a.stop && w >= 0) {  // items are left: a raised flag ends the launch as stopped
                uint32_t st = 0;
                if (lane == 0) st = *a.stop;
                stop = __shfl_sync(FULL, st, 0) != 0;
                if (stop && lane == 0) atomicExch(a.stopped, 1u);
            }
            if (lane == 0) sh.win = stop ? -1 : w;
        }
        __syncthreads();
        const int win = sh.win;
        if (win < 0) break;
        const WinInfo &W = a.win[win];
        if (win != cur) {
            tc_toeplitz<D::N1, D::K1>(b1, W.mu, TC_MU_WORDS, W.mu_off, 4 * D::NT);
            tc_toeplitz<D::N2, D::K2>(b2, W.K, L, 0, 4 * D::NZ);
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            cur = win;
        }
        // fill the CTA's lanes from the window's queue
        const uint32_t s0 = W.side0, n_side = W.nsides;
        const unsigned long long total = (unsigned long long)n_side * kspan;
        bool have = false;
        uint32_t s = 0, k = 0, Y = 0;
        while (true) {
            const unsigned need = __ballot_sync(FULL, !have);
            if (need == 0) break;
            const int leader = __ffs(need) - 1;
            unsigned long long base = 0;
            if ((int)lane == leader) base = atomicAdd(&a.win_next[win], (unsigned long long)__popc(need));
            base = __shfl_sync(FULL, base, leader);
            if (base >= total) break;
            if (!have) {
                const unsigned long long t = base + __popc(need & ((1u << lane) - 1));
                if (t < total) {
                    k = (uint32_t)(t / n_side);
                    s = s0 + (uint32_t)(t - (unsigned long long)k * n_side);
                    have = pick_item(a, s, k, Y);
                }
            }
        }
        // the candidates: n = m*K + X, a1 = m^-1 mod n (both in local memory)
        uint32_t n_loc[L], a_loc[L], y[L];
        uint32_t m = 0, xabs = 0, j = 0;
        int B = 0, sbit = 0;
        double ratio = 0;
        const bool prev = s & 1;
#pragma unroll
        for (int i = 0; i < L; i++) y[i] = 0;
        if (have) {
            m = (uint32_t)a.ms[s >> 1];
            xabs = 2 * Y;
            uint32_t x[L];
            build_candidate<L>(W.K, m, Y, prev, x);
            B = bit_length<L>(x);
            double nd = 0, scale = 1.0;  // n / 2^(32 (NZ-TOP)), NZ - TOP = L - 4
#pragma unroll
            for (int i = 0; i < L; i++) n_loc[i] = x[i];
#pragma unroll
            for (int i = 0; i < L; i++)
                if (!sbit) {
                    const uint32_t word = i ? x[i] : x[i] & ~1u;
                    if (word) sbit = 32 * i + __ffs(word) - 1;
                }
#pragma unroll
            for (int i = L - 1; i >= L - 4; i--) nd = nd * 0x1p32 + (double)x[i];
            for (int i = L - 5; i >= L - 8; i--) {
                scale *= 0x1p-32;
                nd += (double)n_loc[i] * scale;
            }
            ratio = (prev ? (double)xabs : -(double)xabs) / nd;
            if (tc_inverse(m, xabs, prev, j)) {
                tc_start<L>(y, W.K, j, m, prev ? -(int64_t)xabs : (int64_t)xabs, 1, nullptr);
#pragma unroll
                for (int i = 0; i < L; i++) a_loc[i] = y[i];
            } else {  // gcd(m, X) divides n: composite, as by trial division (past sl, where no sieve row rules it out)
                have = false;
                m = xabs = 0;
                ratio = 0;
                B = 0;
            }
        }
        const long long t_round = clock64();
        const int wb = __reduce_max_sync(FULL, B);
        const bool late = __any_sync(FULL, have && sbit > B - 16);
        if (lane == 0) sh.bmax[tid >> 5] = wb | (late ? 1 << 16 : 0);
        if (!__syncthreads_or(have)) continue;  // the window's queue ran out under the CTA
        if (tid == 0 && a.settle) atomicAdd(&a.rounds[0], 1u);
        const int b0 = sh.bmax[0], b1m = sh.bmax[1], b2m = sh.bmax[2], b3 = sh.bmax[3];
        const int bmax = max(max(b0 & 0xffff, b1m & 0xffff), max(b2m & 0xffff, b3 & 0xffff));
        // The exponent's leading bits cost no step: x = 2^e, e = the bits above
        // the low bmax - lead ones, is below K (K > 2^(bmax-32), m < 2^30), and
        // x * m^-1 = s*K + (s*X + 2^e)/m with s = -2^e * X^-1 mod m.  A candidate
        // whose n - 1 ends above those bits would miss a comparison: then lead = 0.
        // Seven to nine steps of 461 .. 1 100 saved: P = 337 2.98 -> 2.94 ms, P = 503
        // 75.9 -> 74.5, P = 811 35.2 -> 34.4; from L = 40 the step itself compiles
        // to a slower one beside it (P = 907 36.2 -> 36.3), so it is left out there.
        const bool early = (b0 | b1m | b2m | b3) >> 16;
        const int lead = L >= 40 || early ? 0 : 31 - __clz(bmax - 32);
        if (have && lead) {
            const int sh0 = bmax - lead, wi = sh0 >> 5;
            const uint32_t lo = n_loc[wi], hi = wi + 1 < L ? n_loc[wi + 1] : 0u;
            const uint32_t e = wi < L ? __funnelshift_r(lo, hi, sh0 & 31) : 0u;
            uint32_t q[L];
            const uint32_t rho = tc_pow2_div<L>(q, e, m);
            const uint32_t sx = (uint32_t)((uint64_t)j * rho % m);
            tc_start<L>(y, W.K, sx, m, prev ? -(int64_t)xabs : (int64_t)xabs, rho, q);
        }
        // y stands for 2^((n-1) >> (b+1)); lanes with fewer bits hold 1 until their top bit
        bool pr = false, done = !have;
        uint32_t ew = have ? n_loc[(bmax - 1 - lead) >> 5] : 0;
        for (int b = bmax - 1 - lead; b >= 0; b--) {
            if (have && (b & 31) == 31) ew = n_loc[b >> 5];
            if (!done && b < sbit) {
                uint32_t c[L];
#pragma unroll
                for (int i = 0; i < L; i++) c[i] = y[i];
                const int r = tc_compare<L>(c, a_loc, n_loc);
                if (r) {  // x = 1 passes only as 2^d (b = s - 1), x = -1 always
                    pr = r == 2 || b == sbit - 1;
                    done = true;
                }
            }
            if (b == 0) break;
            if (!tc_step<L>(S, y, m, xabs, prev ? 0xffffffffu : 0u, ratio, (ew >> (b & 31)) & 1u)) break;
        }
        if (!__syncthreads_and(S.ok)) {
            if (tid == 0) {
                atomicExch(a.failed, 1u);
                // the matrix instruction that was given up on may still read shared
                // memory and write TMEM: once more the limit before both are freed
                tc_wait(S.mbar, S.phase ^ 1u);
            }
            break;
        }
        if (have) {
            ntests++;
            if (pr && atomicMin(&a.found_k[s], k) == NOT_FOUND && a.unresolved) atomicSub(a.unresolved, 1u);
        }
        if (a.settle) {  // wait, within the limit, for the rounds under way (see round_blocks in pg_api.cu)
            __threadfence();
            __syncthreads();
            if (tid == 0) settle_round(a, t_round);
        }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) ntests += __shfl_down_sync(FULL, ntests, o);
    if (lane == 0 && ntests) atomicAdd(a.tests, ntests);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    if (tid < 32)
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(S.tmem), "r"((uint32_t)D::COLS));
}

// ------------------------------------------------------------ launchers

// CTAs of k_search_tc<L> an SM holds: registers, shared memory (1 KB of it per
// CTA is the system's), TMEM columns
template <int L>
int tc_occupancy_t() {
    cudaFuncAttributes at;
    if (cudaFuncGetAttributes(&at, k_search_tc<L>) != cudaSuccess) return 0;
    const int regs = 65536 / ((at.numRegs + 7) / 8 * 8 * TC_ROWS);
    const int smem = 227 * 1024 / (TcDim<L>::SMEM + (int)at.sharedSizeBytes + 1024);
    const int tmem = 512 / TcDim<L>::COLS;
    const int per = regs < smem ? regs : smem;
    return per < tmem ? per : tmem;
}

template <int L>
cudaError_t launch_search_tc_t(const SearchArgs &a, int grid, cudaStream_t st) {
    cudaError_t e = cudaFuncSetAttribute(k_search_tc<L>, cudaFuncAttributeMaxDynamicSharedMemorySize, TcDim<L>::SMEM);
    if (e != cudaSuccess) return e;
    e = cudaFuncSetAttribute(k_search_tc<L>, cudaFuncAttributePreferredSharedMemoryCarveout,
                             cudaSharedmemCarveoutMaxShared);
    if (e != cudaSuccess) return e;
    k_search_tc<L><<<grid, TC_ROWS, TcDim<L>::SMEM, st>>>(a);
    return cudaGetLastError();
}

#define PG_TC_DECLARE(L)                       \
    extern template int tc_occupancy_t<L>();   \
    extern template cudaError_t launch_search_tc_t<L>(const SearchArgs &, int, cudaStream_t);
#define PG_TC_INSTANTIATE(L)            \
    template int tc_occupancy_t<L>();   \
    template cudaError_t launch_search_tc_t<L>(const SearchArgs &, int, cudaStream_t);

}  // namespace pg
