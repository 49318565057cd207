// dr_windows.cu -- the near S1 lookups, window by window of the Mertens table.
//
// A gather from global memory costs the L1 cache one cycle per 128-byte line it touches, and
// away from the end of an S1 range every lane touches its own.  Here a CTA stages a window of
// kTileWin table values in shared memory and sums, over a run of candidate blocks, every
// lookup M(floor(y/n)) whose quotient lies in it: 32 random 2-byte reads of shared memory
// cost about 3.5 cycles of bank conflicts instead of up to 32.  The tile groups, the index
// ranges and the one-FMA quotient are those of dr_tiles.cu; the lookups above a block's last
// window (tile_windows) stay there.  Each lookup is taken by the window q / kTileWin exactly:
// a block of divisors that reaches past the window, for some member, tests every quotient.
// Which (window, block) pairs are looked at is the host's choice (window_items), so the planner
// counts the lookups it leaves to this kernel and the kernel those it sums; a call where they
// differ fails (a count per lane: sums phase 21.07 -> 21.04 ms at 10^16, 97.85 -> 97.93 at 10^17).
//
// Bound: the shared-memory pipe and instruction issue together (1.8 wavefronts per shared
// load, 8.6 instructions per lookup).  M(10^16): 2.6e10 lookups in 11.4 ms, 2.3e12 a second,
// against 0.26e12 (no two lanes on one line) to 2.4e12 from global memory; the sums phase as a
// whole 25.9 -> 21.6 ms, at 10^17 136 -> 101 ms.  Windows of 98304 values by one CTA of 32
// warps; 49152 by two of 16: 22.7 and 112 ms.
//
// Sums: mertens_dr.hpp:1490-1614; streaming M windows: mertens_dr_windowed.hpp:218-374.
#include "dr_kernels.cuh"

#include <algorithm>
#include <cstddef>

namespace drb {

namespace {

constexpr int kWinCta = 1024;
// Union of index ranges below which the lanes take the members and the divisors come in turn
// (with windows down to 32 divisors instead of 64: M(10^17) sums 100.8 -> 98.8 ms).
constexpr uint32_t kNarrow = 48;

struct __align__(16) WinMember {
    double yd;   // y + 1/2
    int32_t sg;  // sign of its terms in this segment
    int32_t pad;
};

struct WinShared {
    WinMember e[kWinCta / 32][32];
    uint2 r[kWinCta / 32][32];  // members' index ranges (blocks past some member's range)
    TileWinTask task;
    uint32_t next;  // the task's next unit
    __align__(16) int16_t win[kTileWin + 8];  // win[7 + i] = M(q0 + i)
};

// M(q) from the staged window: base is the shared address of M(0) if it were staged
// (modulo 2^32), so that the quotient needs no subtraction.  The clobber says that the read
// depends on the staging stores and the barrier after them (it costs nothing: sums phase at
// 10^16 21.07 ms with and without, 21.27 through a C++ pointer with its 64-bit address).
__device__ __forceinline__ int win_M(uint32_t base, uint32_t q) {
    short v;
    asm volatile("ld.shared.s16 %0, [%1];" : "=h"(v) : "r"(base + 2u * q) : "memory");
    return (int)v;
}

// Sum over a block of 128 divisors (4 per lane) and the members [ma, mb), whose ranges the
// block lies in (MASK: meets).
template <bool MASK>
__device__ __forceinline__ int win_block(uint32_t base, const WinMember* E, const uint2* R, const double* r,
                                         uint32_t i0, int ma, int mb, int lane) {
    int s = 0;
#pragma unroll 2
    for (int m = ma; m < mb; ++m) {
        const int4 mv = *reinterpret_cast<const int4*>(E + m);  // one 16-byte read
        const WinMember M{__hiloint2double(mv.y, mv.x), mv.z, 0};
        int v[4];
        if (MASK) {
            const uint2 g = R[m];
#pragma unroll
            for (int p = 0; p < 4; ++p) {
                const uint32_t i = i0 + 32u * p + (uint32_t)lane;
                v[p] = 0;
                if (i >= g.x && i <= g.y) v[p] = win_M(base, floor_q(M.yd, r[p]));
            }
        } else {
#pragma unroll
            for (int p = 0; p < 4; ++p) v[p] = win_M(base, floor_q(M.yd, r[p]));
        }
        s += M.sg * ((v[0] + v[1]) + (v[2] + v[3]));
    }
    return s;
}

// smallest index with divisor >= n, largest with divisor <= n (1 <= n < 2^31; the result of
// the second is below the first index, or -1 as unsigned, where there is none)
__device__ __forceinline__ uint32_t index_from(uint32_t code, uint32_t n, uint32_t res) {
    if (code == 0) return n;
    if (code == 3) {
        const uint32_t i = (n - 1u) / 3u;
        return i + (3u * i + 1u + (i & 1u) < n ? 1u : 0u);
    }
    const uint32_t st = code == 1 ? 2u : 6u;
    return n <= res ? 0u : (n - res + st - 1u) / st;
}
__device__ __forceinline__ int32_t index_to(uint32_t code, uint32_t n, uint32_t res) {
    if (code == 0) return (int32_t)n;
    if (code == 3) {
        const uint32_t i = (n - 1u) / 3u;
        return (int32_t)i - (3u * i + 1u + (i & 1u) > n ? 1 : 0);
    }
    return n < res ? -1 : (int32_t)((n - res) / (code == 1 ? 2u : 6u));
}

__global__ void __launch_bounds__(kWinCta, 1024 / kWinCta) windows_kernel(const TileWinArgs a) {
    extern __shared__ __align__(16) unsigned char win_smem[];
    WinShared& S = *reinterpret_cast<WinShared*>(win_smem);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    WinMember* E = S.e[warp];
    uint2* R = S.r[warp];
    uint32_t cur_w = 0xFFFFFFFFu;
    int cur_q = -1;
    i64 acc = 0;
    uint32_t taken = 0;  // lookups summed by this lane's members, modulo 2^32
    for (;;) {
        __syncthreads();  // every warp is done with the task before and its window
        if (threadIdx.x == 0) {
            const u64 t = atomicAdd(a.ticket, 1ull);
            S.task = t < a.n_tasks ? a.tasks[t] : TileWinTask{0xFFFFFFFFu, 0u, 0u, 0u};
            S.next = 0;
        }
        __syncthreads();
        const TileWinTask I = S.task;
        if (I.w == 0xFFFFFFFFu) break;
        const u64 q0 = (u64)I.w * kTileWin;
        if (I.w != cur_w) {
            if (I.w > 0) {
                const uint4* src = reinterpret_cast<const uint4*>(a.T.dM + (q0 - 8));
                uint4* dst = reinterpret_cast<uint4*>(S.win);
                for (int t = threadIdx.x; t < (kTileWin + 8) / 8; t += kWinCta) dst[t] = __ldg(src + t);
            } else {
                for (int t = threadIdx.x; t < kTileWin + 8; t += kWinCta)
                    S.win[t] = t >= 8 ? __ldg(a.T.dM + (t - 8)) : (int16_t)0;
            }
            cur_w = I.w;
            __syncthreads();
        }
        const uint32_t base = (uint32_t)__cvta_generic_to_shared(S.win + 7) - 2u * (uint32_t)q0;
        // RN(1/q0), RN(1/q1): floor(y/q) by the same FMA as floor(y/n)
        const double rq0 = q0 ? 1.0 / (double)q0 : 0.0, rq1 = 1.0 / (double)(q0 + kTileWin);
        TileWinItem J = a.items[I.i0];
        uint32_t it = I.i0, u_end = 0;  // the warp's item, and the unit it ends at
        const QueryDev* Q = nullptr;
        const SlotDesc* slots = nullptr;
        u64 blk_base = 0;
        for (;;) {
            uint32_t u = 0;
            if (lane == 0) u = atomicAdd(&S.next, 1u);
            u = __shfl_sync(0xffffffffu, u, 0);
            if (u >= I.units) break;
            if (u >= u_end) {
                while (it + 1 < I.i1 && __ldg(&a.items[it + 1].u0) <= u) ++it;
                J = a.items[it];
                u_end = J.u0 + 2u * (J.b1 - J.b0) * J.parts;
                Q = a.queries + J.q;
                slots = a.slots + __ldg(&Q->slot_base);
                blk_base = __ldg(&Q->blk_base);
                if ((int)J.q != cur_q) {
                    if (cur_q >= 0) {
                        const u64 t = warp_sum_u64((u64)acc);
                        if (lane == 0) atomicAdd(a.acc + 3 * cur_q + 1, t);
                    }
                    acc = 0;
                    cur_q = (int)J.q;
                }
            }
            const uint32_t gi = (u - J.u0) / J.parts, step = J.parts, mine = (u - J.u0) - gi * J.parts;
            const u64 gid = 2ull * J.b0 + gi;
            const WinGroup* G = a.groups + gid;
            if (__ldg(&G->wc) <= I.w) continue;
            const uint32_t mm = __ldg(&G->mm), bits = __ldg(&G->bits);
            const bool member = (mm >> lane) & 1u;
            const int rank = __popc(mm & ((1u << lane) - 1u));
            const SlotDesc* d = slots + (2 * (32 * ((gid >> 1) - blk_base) + (u64)(member ? lane : __ffs(mm) - 1)) +
                                         (gid & 1));
            const double yd = (double)(i64)__ldg(&d->y) + 0.5;
            // this member's divisors with a quotient in the window, [nlo, nhi]
            const u64 na = ((u64)__double_as_longlong(__fma_rd(yd, rq1, 4503599627370496.0)) & 0xFFFFFFFFFFFFFull) + 1;
            const u64 nb = q0 ? (u64)__double_as_longlong(__fma_rd(yd, rq0, 4503599627370496.0)) & 0xFFFFFFFFFFFFFull
                              : 0x7FFFFFF0ull;
            const uint32_t nlo = (uint32_t)min(na, (u64)0x7FFFFFF1u), nhi = (uint32_t)min(nb, (u64)0x7FFFFFF0u);
            const uint32_t nmin = __reduce_min_sync(0xffffffffu, nlo), nmax = __reduce_max_sync(0xffffffffu, nhi);
            if (nmin > nmax || nmax == 0) continue;
            const uint32_t dbits = (uint32_t)__ldg(&d->bits);
            __syncwarp();
            if (member) E[rank].yd = yd;
#pragma unroll 1
            for (int g = 0; g < kS1Seg; ++g) {
                const uint32_t ulo = __ldg(&G->ulo[g]), uhi = __ldg(&G->uhi[g]);
                const uint32_t code = (bits >> (3 + 3 * g)) & 3u;
                const uint32_t div = code == 0 ? 1u : code == 1 ? 2u : code == 2 ? 6u : 3u;
                if (ulo > uhi || nmax / div + 1u < ulo || nmin > div * uhi + 6u) continue;
                // the member's part of the segment
                const u64 cnt2 = (u64)__ldg(&d->cnt[g]);
                const uint32_t cnt = (uint32_t)cnt2 + (uint32_t)(cnt2 >> 32), n0 = (uint32_t)__ldg(&d->n0[g]);
                uint32_t lo = code == 1 ? n0 >> 1 : code == 2 ? n0 / 6u : n0;
                uint32_t res = code == 1 ? n0 & 1u : code == 2 ? n0 % 6u : 0u;
                int32_t hi = (int32_t)(lo + cnt) - 1;
                bool some = member && cnt > 0 && nlo <= nhi && nhi > 0;
                if (some) {
                    lo = max(lo, index_from(code, nlo, res));
                    hi = min(hi, index_to(code, nhi, res));
                    some = (int32_t)lo <= hi;
                }
                const uint32_t umin = __reduce_min_sync(0xffffffffu, some ? lo : 0xffffffffu);
                const uint32_t umax = __reduce_max_sync(0xffffffffu, some ? (uint32_t)hi : 0u);
                if (umin > umax) continue;
                res = __reduce_max_sync(0xffffffffu, member && cnt > 0 ? res : 0u);
                const uint32_t tot = __reduce_add_sync(0xffffffffu, some ? (uint32_t)hi - lo + 1u : 0u);
                if (mine == 0 && some) taken += (uint32_t)hi - lo + 1u;
                const int sgn = ((dbits >> 2) & 1u) == ((dbits >> (5 + 3 * g)) & 1u) ? 1 : -1;
                if (umax - umin < kNarrow) {
                    // few divisors, all members at once: lanes on members, the divisors in turn
                    double* rs = reinterpret_cast<double*>(R);
                    int part = 0;
                    for (uint32_t c = mine; 32u * c <= umax - umin; c += step) {
                        const uint32_t i0 = umin + 32u * c;
                        __syncwarp();
                        rs[lane] = __ldg(a.rcp + tile_n(code, min(i0 + (uint32_t)lane, umax), res));
                        __syncwarp();
                        const int cnt = (int)min(32u, umax - i0 + 1u);
#pragma unroll 4
                        for (int t = 0; t < cnt; ++t) {
                            const uint32_t i = i0 + (uint32_t)t;
                            if (some && i >= lo && i <= (uint32_t)hi) part += win_M(base, floor_q(yd, rs[t]));
                        }
                    }
                    acc += (i64)(sgn * part);
                    __syncwarp();
                    continue;
                }
                __syncwarp();
                if (member) {
                    E[rank].sg = sgn;
                    R[rank] = some ? make_uint2(lo, (uint32_t)hi) : make_uint2(1u, 0u);
                }
                __syncwarp();
                if (tot / 4u >= umax - umin) {
                    // the members' ranges overlap: blocks of divisors over their union
                    const uint32_t nblk = (umax - umin) / kTileN + 1u;
                    for (uint32_t bi = mine; bi < nblk; bi += step) {
                        const uint32_t i0 = umin + kTileN * bi, i1 = i0 + (kTileN - 1);
                        const unsigned act = __ballot_sync(0xffffffffu, some && lo <= i1 && (uint32_t)hi >= i0);
                        if (act == 0) continue;
                        const unsigned whole = __ballot_sync(0xffffffffu, some && lo <= i0 && (uint32_t)hi >= i1);
                        const int ma = __popc(mm & ((act & -act) - 1u)), mb = __popc(mm & (~0u >> __clz(act)));
                        double r[4];
#pragma unroll
                        for (int p = 0; p < 4; ++p)
                            r[p] = __ldg(a.rcp + tile_n(code, min(i0 + 32u * p + (uint32_t)lane, umax), res));
                        if (__popc(whole) == mb - ma) acc += win_block<false>(base, E, R, r, i0, ma, mb, lane);
                        else acc += win_block<true>(base, E, R, r, i0, ma, mb, lane);
                    }
                } else {
                    // few members at a time: one after another.  `part` fits 32 bits: `parts` is
                    // cut so that a unit holds about 131072 lookups by the estimate of window_items,
                    // which is never below one member's share, and where it stops at 1024 pieces a
                    // lane's share of the divisors, below 2^31, is at most 2^16 of |M| < 27000.
                    unsigned left = __ballot_sync(0xffffffffu, some);
                    while (left) {
                        const int m = __popc(mm & ((left & -left) - 1u));
                        left &= left - 1u;
                        const uint2 g2 = R[m];
                        const double yd1 = E[m].yd;
                        int part = 0;
                        for (uint32_t i0 = g2.x + 256u * ((mine + (uint32_t)m) % step); i0 <= g2.y; i0 += 256u * step) {
                            double r[8];
                            int v[8];
#pragma unroll
                            for (int p = 0; p < 8; ++p)
                                r[p] = __ldg(a.rcp + tile_n(code, min(i0 + 32u * p + (uint32_t)lane, g2.y), res));
#pragma unroll
                            for (int p = 0; p < 8; ++p) v[p] = win_M(base, floor_q(yd1, r[p]));
#pragma unroll
                            for (int p = 0; p < 8; ++p) part += i0 + 32u * p + (uint32_t)lane <= g2.y ? v[p] : 0;
                        }
                        acc += (i64)(E[m].sg * part);
                    }
                }
            }
        }
    }
    if (cur_q >= 0) {
        const u64 t = warp_sum_u64((u64)acc);
        if (lane == 0) atomicAdd(a.acc + 3 * cur_q + 1, t);
    }
    taken = __reduce_add_sync(0xffffffffu, taken);
    if (lane == 0) atomicAdd(reinterpret_cast<uint32_t*>(a.ticket + 1), 0u - taken);
}

static_assert(offsetof(WinShared, win) % 16 == 0 && kTileWin % 8 == 0, "16-byte staging copies");

}  // namespace

void launch_windows(const TileWinArgs& a, int sm_count, cudaStream_t s) {
    if (a.n_tasks == 0) return;
    cudaFuncSetAttribute(windows_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(WinShared));
    const int grid = (int)std::min<u64>(a.n_tasks, (u64)sm_count * (1024 / kWinCta));
    windows_kernel<<<grid, kWinCta, sizeof(WinShared), s>>>(a);
}

}  // namespace drb
