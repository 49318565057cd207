// dr_tiles.cu -- the S1/S2 sums over tiles of (evaluations x divisors).
//
// The evaluations of neighbouring candidates k walk nearly the same divisors n (S1) and
// wheel positions j (S2).  A tile group (dr_device.cuh) holds up to 32 of them; a work
// unit is one block of 128 divisors or 64 wheel positions for all members whose range
// meets it, so that the reciprocal and mu(j) of a divisor are read once per group instead
// of once per evaluation.  y falls along a group and the ranges with it, so those members
// are neighbours: [ma, mb) below.
//
// Exact quotients from one instruction.  For y < 2^51 and r = RN(1/n) the product
// (y + 1/2) * r lies strictly between floor(y/n) and floor(y/n) + 1: (y + 1/2)/n is at
// least 1/(2n) away from both, and r's relative error of 2^-53 moves it by less than
// (2^51 + 1)/n * 2^-53 < 1/(2n).  y + 1/2 is exact in FP64, so an FMA rounded down,
// RD((y + 1/2) * r + 2^52), is 2^52 + floor(y/n): the low mantissa word is the quotient
// itself, with no integer correction (cf. fast_div, mertens_dr.hpp:80-86).
//
// Bound: S1 by the L1 cache's tag and data stages (a warp gather costs one cycle per
// 128-byte line it touches: 1 lookup per cycle and SM where all lanes differ, about 9 where
// neighbouring quotients share lines), S2 by instruction issue.  Sums phase on B200, one
// evaluation at a time -> tiles: M(10^15), reference parameters 10.0 -> 5.3 ms; M(10^16)
// 48.6 -> 25.9 ms and M(10^17) 261 -> 136 ms at the B200 policy; M(10^12) 0.42 -> 0.16 ms
// (dense table).  Two CTAs of 8 warps per SM (128 registers, no spills) beat three (80) and
// four (64): 28.9, 29.0, 31.5 ms at M(10^16).
//
// Launches of little work or of few candidates stay with the sums kernel (tiles_pay, dr_engine.cpp).
//
// Sums: mertens_dr.hpp:1490-1614 (S1), :462-660 (S2).
#include "dr_kernels.cuh"

#include <algorithm>

namespace drb {

namespace {

constexpr int kTileWarps = 8;           // warps per CTA
constexpr double kTwo52 = 4503599627370496.0;

struct __align__(16) TileMember {
    double yd;   // y + 1/2
    int32_t sg;  // sign of the evaluation's terms in this segment (0: none)
    int32_t pad;
};

// one 16-byte read (left to itself the compiler reads yd and sg separately)
__device__ __forceinline__ TileMember member_of(const TileMember* p) {
    const int4 v = *reinterpret_cast<const int4*>(p);
    return TileMember{__hiloint2double(v.y, v.x), v.z, 0};
}

// One warp's state: the members of the group and, where a block reaches past the range of
// some member, their ranges (S1: index range, S2: j range).
struct TileWarp {
    TileMember e[34];
    uint2 r[34];
    double rcp[kTileN];
};

// exact double of a 32-bit integer on the FP64 pipe (the conversions run on a narrower one)
__device__ __forceinline__ double u32_double(uint32_t v) {
    return __hiloint2double(0x43300000, (int)v) - kTwo52;
}

__device__ __forceinline__ u64 floor_q64(double yd, double r) {
    return (u64)__double_as_longlong(__fma_rd(yd, r, kTwo52)) & 0xFFFFFFFFFFFFFull;
}

// largest s in [0, n_slots) with prefix[s] <= o, by the whole warp (32-way search)
__device__ __forceinline__ u64 warp_upper_slot(const u64* prefix, u64 n_slots, u64 o, int lane) {
    u64 lo = 0, hi = n_slots - 1;
    while (lo < hi) {
        const u64 step = (hi - lo) / 32 + 1;
        const u64 at = lo + step * (u64)lane;
        const unsigned le = __ballot_sync(0xffffffffu, at <= hi && prefix[at] <= o);
        const u64 base = lo + step * (u64)(__popc(le) - 1);  // lane 0 always holds
        hi = min(hi, base + step - 1);
        lo = base;
    }
    return lo;
}

// S1, lanes on divisors: 4 divisors per lane, members one after another, every quotient in
// the dense tier.  MASK: a member's divisors outside its own range are left out.
template <bool MASK>
__device__ __forceinline__ int s1_lanes_n(const int16_t* dMm1, const TileWarp& W, const double* r, uint32_t i0,
                                          int ma, int mb, int lane) {
    int s = 0;
#pragma unroll 2
    for (int m = ma; m < mb; ++m) {
        const TileMember E = member_of(&W.e[m]);
        int v[4];
        if (MASK) {
            const uint2 R = W.r[m];
#pragma unroll
            for (int p = 0; p < 4; ++p) {
                const uint32_t i = i0 + 32u * p + (uint32_t)lane;
                v[p] = 0;
                if (i >= R.x && i <= R.y) v[p] = __ldg(dMm1 + floor_q(E.yd, r[p]));
            }
        } else {
#pragma unroll
            for (int p = 0; p < 4; ++p) v[p] = __ldg(dMm1 + floor_q(E.yd, r[p]));
        }
        s += E.sg * ((v[0] + v[1]) + (v[2] + v[3]));
    }
    return s;
}

// S1, lanes on members: the block's divisors one after another (reciprocals staged in
// shared memory).  Every member's range holds the whole block.
__device__ __forceinline__ int s1_lanes_k(const int16_t* dMm1, const TileWarp& W, int ma, int mb, int lane) {
    const TileMember E = W.e[ma + lane < mb ? ma + lane : ma];
    int s = 0;
#pragma unroll 2
    for (int i = 0; i < (int)kTileN; i += 8) {
        int v[8];
#pragma unroll
        for (int p = 0; p < 8; p += 2) {
            const double2 r = *reinterpret_cast<const double2*>(&W.rcp[i + p]);
            v[p] = __ldg(dMm1 + floor_q(E.yd, r.x));
            v[p + 1] = __ldg(dMm1 + floor_q(E.yd, r.y));
        }
#pragma unroll
        for (int p = 0; p < 8; ++p) s += v[p];
    }
    return ma + lane < mb ? s * E.sg : 0;
}

// S1, any quotient (compressed tier, or beyond 32 bits)
__device__ __noinline__ i64 s1_any(const SumsArgs& a, const TileWarp& W, uint32_t code, uint32_t res, uint32_t i0,
                                   int ma, int mb, int lane) {
    double r[4];
#pragma unroll
    for (int p = 0; p < 4; ++p) {
        const uint32_t n = tile_n(code, i0 + 32u * p + (uint32_t)lane, res);
        r[p] = n <= a.inv_limit ? __ldg(a.rcp + n) : 0.0;  // 0: past every member's range
    }
    i64 s = 0;
#pragma unroll 2
    for (int m = ma; m < mb; ++m) {
        const uint2 R = W.r[m];
        int32_t v[4];
#pragma unroll
        for (int p = 0; p < 4; ++p) {
            const uint32_t i = i0 + 32u * p + (uint32_t)lane;
            v[p] = i >= R.x && i <= R.y ? table_M(a.T, floor_q64(W.e[m].yd, r[p])) : 0;
        }
        s += (i64)W.e[m].sg * (((i64)v[0] + v[1]) + ((i64)v[2] + v[3]));
    }
    return s;
}

// S2 on two wheel positions per lane, i.e. four j: j[c], r[c] = RN(1/j[c]), mu[c].  Per
// member and j one quotient and the summand's parts, summed over the members in 32 bits
// (every quotient below 2^26) or, WIDE, in 64 (below 2^31), and times mu(j) once at the
// end.  Kinds as in sums_kernel:
//   1: q   2: (q+1)/2 = (q + (q&1))/2   3: q & 1   4: q/4 + (q&1)   0: a*(q/12) + T[q mod 12]
// The parities are collected as bits, one per member, and counted against the members'
// signs afterwards.
template <bool WIDE>
struct TileAcc {
    typedef int32_t type;
};
template <>
struct TileAcc<true> {
    typedef i64 type;
};

template <int KIND, bool MASK, bool WIDE>
__device__ __forceinline__ i64 s2_tile(const TileWarp& W, const int32_t* sT, int32_t a12, const uint32_t* j,
                                       const double* r, const int32_t* mu, int ma, int mb, uint32_t pos,
                                       uint32_t neg, bool exact) {
    typedef typename TileAcc<WIDE>::type A;
    A acc[4] = {0, 0, 0, 0};
    int32_t t[4] = {0, 0, 0, 0};
    uint32_t par[4] = {0, 0, 0, 0};
    double r12[4];
    if (KIND == 0) {
#pragma unroll
        for (int c = 0; c < 4; ++c) r12[c] = r[c] * (1.0 / 12.0);
        if (exact) {  // RN(1/(12 j)) to the last bit or so: one Newton step
#pragma unroll
            for (int c = 0; c < 4; ++c)
                r12[c] = __fma_rn(r12[c], __fma_rn(-12.0 * u32_double(j[c]), r12[c], 1.0), r12[c]);
        }
    }
#pragma unroll(MASK || KIND == 0 ? 1 : 2)
    for (int m = ma; m < mb; ++m) {
        const TileMember E = member_of(&W.e[m]);
        uint2 R = make_uint2(0u, 0u);
        if (MASK) R = W.r[m];
#pragma unroll
        for (int c = 0; c < 4; ++c) {
            uint32_t q = floor_q(E.yd, r[c]);
            const bool out = MASK && (j[c] < R.x || j[c] > R.y);
            if (MASK) q = out ? 0u : q;
            if (KIND == 1 || KIND == 2) acc[c] += (A)E.sg * (A)(int32_t)q;
            if (KIND == 4) acc[c] += (A)E.sg * (A)(int32_t)(q >> 2);
            if (KIND >= 2) par[c] = __funnelshift_r(par[c], q, 1);  // bit 31 = parity of q
            if (KIND == 0) {
                uint32_t k = floor_q(E.yd, r12[c]);
                if (MASK) k = out ? 0u : k;
                acc[c] += (A)E.sg * (A)(int32_t)k;
                t[c] += E.sg * sT[q - 12u * k];
            }
        }
    }
    i64 s = 0;
#pragma unroll
    for (int c = 0; c < 4; ++c) {
        const int32_t p = KIND >= 2 ? __popc(par[c] & pos) - __popc(par[c] & neg) : 0;
        A v;  // every summand is at most its quotient: the sum fits A as the quotients' does
        if (KIND == 1) v = acc[c];
        else if (KIND == 2) v = (acc[c] + p) >> 1;  // an even sum
        else if (KIND == 3) v = p;
        else if (KIND == 4) v = acc[c] + p;
        else v = (A)a12 * acc[c] + t[c];
        s += (i64)mu[c] * (i64)v;
    }
    return s;
}

// mu(j) and 1/j of the two j of wheel position m, j[0] = 6m+1 and j[1] = 6m+5.  invw's
// reciprocals are up to 3.5 ulp off (mu in the low bits), which leaves (y + 1/2) r between the
// same two integers while y < 2^48 (2^48 * 7 * 2^-53 < 1/2, and r/12 adds two roundings:
// 2^48 * 9 * 2^-53 < 1/2).  Above (`exact`), one Newton step brings them to within 2^-53
// (1 + 2^-40) of 1/j.
constexpr double kExactRcpY = 281474976710656.0;  // 2^48
__device__ __forceinline__ void wheel_pair(const double2 iv, uint32_t m, double* r, int32_t* mu, bool exact) {
    r[0] = iv.x;
    r[1] = iv.y;
    if (exact) {
        r[0] = __fma_rn(iv.x, __fma_rn(-u32_double(6u * m + 1u), iv.x, 1.0), iv.x);
        r[1] = __fma_rn(iv.y, __fma_rn(-u32_double(6u * m + 5u), iv.y, 1.0), iv.y);
    }
    mu[0] = (int32_t)((uint32_t)__double2loint(iv.x) << 30) >> 30;
    mu[1] = (int32_t)((uint32_t)__double2loint(iv.y) << 30) >> 30;
}

// S2, quotients of 2^31 and above
__device__ __noinline__ i64 s2_any(const SumsArgs& a, const TileWarp& W, const int32_t* sT, int32_t a12, uint32_t m0,
                                   uint32_t mmax, int ma, int mb, int lane) {
    i64 s = 0;
    for (uint32_t m = m0 + (uint32_t)lane; m < m0 + kTileM && m <= mmax; m += 32) {
        double r[2];
        int32_t mu[2];
        wheel_pair(__ldg(a.invw + m), m, r, mu, true);
        for (int h = 0; h < 2; ++h) {
            const uint32_t j = 6u * m + (h ? 5u : 1u);
            const double rj = h ? r[1] : r[0];
            for (int e = ma; e < mb; ++e) {
                const uint2 R = W.r[e];
                if (j < R.x || j > R.y) continue;
                const u64 q = floor_q64(W.e[e].yd, rj);
                const u64 k = q / 12u;
                s += (i64)(W.e[e].sg * (h ? mu[1] : mu[0])) * ((i64)a12 * (i64)k + sT[q - 12u * k]);
            }
        }
    }
    return s;
}

template <int KIND>
__device__ __forceinline__ i64 s2_block(const TileWarp& W, const int32_t* sT, int32_t a12, const uint32_t* j,
                                        const double* r, const int32_t* mu, int ma, int mb, uint32_t pos,
                                        uint32_t neg, bool core, bool wide, bool exact) {
    if (wide) return s2_tile<KIND, true, true>(W, sT, a12, j, r, mu, ma, mb, pos, neg, exact);
    if (core) return s2_tile<KIND, false, false>(W, sT, a12, j, r, mu, ma, mb, pos, neg, exact);
    return s2_tile<KIND, true, false>(W, sT, a12, j, r, mu, ma, mb, pos, neg, exact);
}

// kind of piece 1..12 (piece_kind of sums_kernel)
__device__ __forceinline__ int tile_kind(int piece) {
    return piece == 8 || piece == 12 ? 1 : piece == 7 || piece == 11 ? 2 : piece == 6 ? 3 : piece == 5 ? 4 : 0;
}


__global__ void __launch_bounds__(32 * kTileWarps, 2) tiles_kernel(const SumsArgs a) {
    __shared__ TileWarp sw[kTileWarps];
    __shared__ int32_t sT[13 * 12];  // piece(r) for r < 12, every piece
    for (int t = threadIdx.x; t < 13 * 12; t += blockDim.x) sT[t] = (int32_t)piece_formula(t / 12, t % 12);
    __syncthreads();
    const int lane = threadIdx.x & 31;
    TileWarp& W = sw[threadIdx.x >> 5];
    const int16_t* dMm1 = a.T.dM - 1;  // dMm1[q] = M(q)
    const double dense_q = (double)min(a.T.u_dense, (i64)0xFFFFFFFEll);
    const u64 n_groups = 2 * a.n_blocks, total = a.prefix[n_groups];
    // Units per ticket: neighbouring units of a group share its set-up and table lines in L1,
    // so up to 64 (32: 2% more at M(10^16), 4% at the 256-query batch), but 16 tickets per warp
    // so that the last ones do not wait for one long one (8 tickets of up to 128: 2.0 -> 2.5 ms
    // at M(2 * 10^14)).
    u64 per = a.chunk_log2 > 0 ? 1ull << max(0, min(a.chunk_log2 - 12, 5)) : 0ull;  // a unit: about 2^12 ops
    if (per == 0) per = max((u64)4, min(total / ((u64)gridDim.x * kTileWarps * 16), (u64)64));
    int cur_q = -1;
    u64 s1 = 0, s2 = 0;
    for (;;) {
        u64 chunk = 0;
        if (lane == 0) chunk = atomicAdd(a.ticket, 1ull);
        chunk = __shfl_sync(0xffffffffu, chunk, 0);
        u64 o = chunk * per;
        if (o >= total) break;
        const u64 o_end = min(o + per, total);
        while (o < o_end) {
            const u64 w = warp_upper_slot(a.prefix, n_groups, o, lane);
            const u64 sbase = a.prefix[w], send = a.prefix[w + 1];
            const TileGroup* rec = a.tgroups + w;
            const bool single = __ldg(&rec->single) != 0;
            uint32_t rend = 0, rlo = 1, rhi = 0;
            if (lane < kS1Seg + 8) rend = __ldg(rec->end + lane), rlo = __ldg(rec->lo + lane), rhi = __ldg(rec->hi + lane);
            int qi = 0;
            if (a.nq > 1) {
                int lo = 0, hi = a.nq - 1;
                while (lo < hi) {
                    const int mid = (lo + hi + 1) >> 1;
                    if (a.queries[mid].blk_base <= w >> 1) lo = mid;
                    else hi = mid - 1;
                }
                qi = lo;
            }
            if (qi != cur_q) {
                if (cur_q >= 0) {
                    const u64 t1 = warp_sum_u64(s1), t2 = warp_sum_u64(s2);
                    if (lane == 0) {
                        atomicAdd(a.acc + 3 * cur_q + 1, t1);
                        atomicAdd(a.acc + 3 * cur_q + 2, t2);
                    }
                }
                s1 = s2 = 0;
                cur_q = qi;
            }
            // the block's evaluations, one per lane
            const u64 slot_base = a.queries[qi].slot_base;
            const u64 c = 32 * ((w >> 1) - a.queries[qi].blk_base) + (u64)lane;
            const SlotDesc* mine = a.slots + (slot_base + 2 * c + (w & 1));
            const bool there = c < (u64)a.queries[qi].nc;
            const u64 bits = there ? mine->bits : 0ull;
            const double y_own = there ? (double)(i64)mine->y + 0.5 : 0.0;
            unsigned left = __ballot_sync(0xffffffffu, (bits & kSlotTile) != 0);
            const u64 u0 = o - sbase, u1 = min(o_end, send) - sbase;  // this ticket's units
            const uint32_t rstart = __shfl_up_sync(0xffffffffu, rend, 1);
            const unsigned visit = __ballot_sync(0xffffffffu, lane < kS1Seg + 8 && rend > u0 &&
                                                                  (lane == 0 ? 0u : rstart) < u1);
            u64 useg = 0;
            while (left && useg < u1) {
            const u64 sig = __shfl_sync(0xffffffffu, bits & (kSlotTile | kTileSig), __ffs(left) - 1);
            const bool member = (bits & (kSlotTile | kTileSig)) == sig;
            const unsigned mm = __ballot_sync(0xffffffffu, member);
            left &= ~mm;
            const int rank = __popc(mm & ((1u << lane) - 1u));
            const double yd = member ? y_own : 0.0;
            const uint32_t kbits = (uint32_t)sig;
            const int piece0 = (kbits & 3u) == EVAL_SINGLE ? 9 : 1;
            for (unsigned gm = single ? visit : (1u << (kS1Seg + 8)) - 1u; gm; gm &= gm - 1u) {
                const int g = __ffs(gm) - 1;
                uint32_t lo = 1, hi = 0, res = 0;
                uint2 jr = make_uint2(1u, 0u);
                if (member) tile_range(*mine, g, &lo, &hi, &res, &jr);
                const bool some = lo <= hi;
                uint32_t ulo, uhi;
                u64 ub;
                if (single) {
                    ulo = __shfl_sync(0xffffffffu, rlo, g);
                    uhi = __shfl_sync(0xffffffffu, rhi, g);
                    useg = __shfl_sync(0xffffffffu, rend, g);
                    const uint32_t start = __shfl_sync(0xffffffffu, rstart, g);
                    ub = g ? start : 0u;
                } else {
                    ulo = __reduce_min_sync(0xffffffffu, some ? lo : 0xffffffffu);
                    uhi = __reduce_max_sync(0xffffffffu, some ? hi : 0u);
                    ub = useg;
                    useg += tile_units(g, ulo, uhi);
                }
                const u64 a0 = max(u0, ub), a1 = min(u1, useg);
                if (a0 >= a1) continue;
                const bool plus = !(bits & 4u);
                const bool gplus = g >= kS1Seg || !((bits >> (3 + 3 * g)) & 4u);
                const int sgn = plus == gplus ? 1 : -1;
                __syncwarp();
                if (member) {
                    W.e[rank].yd = yd;
                    W.e[rank].sg = some ? sgn : 0;
                    W.r[rank] = g < kS1Seg ? make_uint2(lo, hi) : jr;
                }
                __syncwarp();
                if (g < kS1Seg) {
                    const uint32_t code = (kbits >> (3 + 3 * g)) & 3u;
                    res = __reduce_max_sync(0xffffffffu, some ? res : 0u);
                    const double span = code == 0 ? 32.0 : code == 1 ? 64.0 : code == 2 ? 192.0 : 96.0;
                    // blocks whose first unit is the ticket's
                    const uint32_t b0 = ((uint32_t)(a0 - ub) + kTileS1Units - 1u) / kTileS1Units;
                    const uint32_t b1 = ((uint32_t)(a1 - ub) + kTileS1Units - 1u) / kTileS1Units;
                    for (uint32_t blk = b0; blk < b1; ++blk) {
                        const uint32_t i0 = ulo + kTileN * blk, i1 = i0 + (kTileN - 1);
                        const unsigned act = __ballot_sync(0xffffffffu, some && lo <= i1 && hi >= i0);
                        const unsigned whole = __ballot_sync(0xffffffffu, some && lo <= i0 && hi >= i1);
                        if (act == 0) continue;
                        int ma = __popc(mm & ((act & -act) - 1u));
                        const int mb = __popc(mm & (~0u >> __clz(act)));
                        bool core = __popc(whole) == mb - ma;
                        const double n0 = (double)tile_n(code, i0, res);
                        // the first members' largest quotients may lie above the dense tier
                        const unsigned far = __ballot_sync(0xffffffffu, member && yd >= dense_q * n0);
                        const int mf = min(mb, __popc(far));
                        if (mf > ma) {
                            s1 += (u64)s1_any(a, W, code, res, i0, ma, mf, lane);
                            if (mf == mb) continue;
                            ma = mf;
                            core = false;
                        }
                        const double y_hi = W.e[ma].yd;
                        double r[4];
#pragma unroll
                        for (int p = 0; p < 4; ++p)
                            r[p] = __ldg(a.rcp + tile_n(code, min(i0 + 32u * p + (uint32_t)lane, uhi), res));
                        if (!core) {
                            s1 += (u64)(i64)s1_lanes_n<true>(dMm1, W, r, i0, ma, mb, lane);
                        } else if (mb - ma >= 16 && (y_hi - W.e[mb - 1].yd) * n0 < y_hi * span) {
                            // the quotients of one divisor lie closer together than those of
                            // 32 neighbouring divisors: fewer table lines per warp load
                            __syncwarp();
#pragma unroll
                            for (int p = 0; p < 4; ++p) W.rcp[32 * p + lane] = r[p];
                            __syncwarp();
                            s1 += (u64)(i64)s1_lanes_k(dMm1, W, ma, mb, lane);
                        } else {
                            s1 += (u64)(i64)s1_lanes_n<false>(dMm1, W, r, i0, ma, mb, lane);
                        }
                    }
                } else {
                    const int piece = piece0 + g - kS1Seg;
                    const int kind = tile_kind(piece);
                    const int32_t* T = sT + 12 * piece;
                    const int32_t a12 = (int32_t)piece_formula(piece, 12);
                    const uint32_t rpos = __reduce_or_sync(0xffffffffu, some && sgn > 0 ? 1u << rank : 0u);
                    const uint32_t rneg = __reduce_or_sync(0xffffffffu, some && sgn < 0 ? 1u << rank : 0u);
                    for (u64 u = a0; u < a1; ++u) {
                        const uint32_t m0 = (ulo & ~31u) + kTileM * (uint32_t)(u - ub);
                        const uint32_t j0 = 6u * m0 + 1u, j1 = 6u * (m0 + kTileM) - 1u;
                        const unsigned act = __ballot_sync(0xffffffffu, some && jr.x <= j1 && jr.y >= j0);
                        const unsigned whole = __ballot_sync(0xffffffffu, some && jr.x <= j0 && jr.y >= j1);
                        if (act == 0) continue;
                        const int ma = __popc(mm & ((act & -act) - 1u)), mb = __popc(mm & (~0u >> __clz(act)));
                        const bool core = __popc(whole) == mb - ma;
                        const double jf = (double)j0, y_hi = W.e[ma].yd;
                        if (!(y_hi < 2147483647.0 * jf)) {
                            s2 += (u64)s2_any(a, W, T, a12, m0, uhi, ma, mb, lane);
                            continue;
                        }
                        const bool exact = !(y_hi < kExactRcpY);
                        uint32_t j[4];
                        double r[4];
                        int32_t mu[4];
#pragma unroll
                        for (int p = 0; p < 2; ++p) {
                            const uint32_t m = m0 + 32u * p + (uint32_t)lane;
                            wheel_pair(__ldg(a.invw + min(m, uhi)), min(m, uhi), r + 2 * p, mu + 2 * p, exact);
                            j[2 * p] = 6u * m + 1u;  // past uhi: outside every member's range
                            j[2 * p + 1] = 6u * m + 5u;
                        }
                        const bool wide = !(y_hi < 67108863.0 * jf);
                        // after mb - ma shifts the parity of member m is bit 32 - mb + m
                        const uint32_t pos = (rpos >> ma) << (32 - (mb - ma)), neg = (rneg >> ma) << (32 - (mb - ma));
                        i64 v;
                        switch (kind) {
                        case 1: v = s2_block<1>(W, T, a12, j, r, mu, ma, mb, pos, neg, core, wide, exact); break;
                        case 2: v = s2_block<2>(W, T, a12, j, r, mu, ma, mb, pos, neg, core, wide, exact); break;
                        case 3: v = s2_block<3>(W, T, a12, j, r, mu, ma, mb, pos, neg, core, wide, exact); break;
                        case 4: v = s2_block<4>(W, T, a12, j, r, mu, ma, mb, pos, neg, core, wide, exact); break;
                        default: v = s2_block<0>(W, T, a12, j, r, mu, ma, mb, pos, neg, core, wide, exact); break;
                        }
                        s2 += (u64)v;
                    }
                }
            }
            }
            if (useg < u1) {
                // planning and this kernel disagree on the group's units: flag it and go on
                if (lane == 0) atomicOr(a.ticket + 1, 1ull);
                break;
            }
            o = sbase + u1;
        }
    }
    if (cur_q >= 0) {
        const u64 t1 = warp_sum_u64(s1), t2 = warp_sum_u64(s2);
        if (lane == 0) {
            atomicAdd(a.acc + 3 * cur_q + 1, t1);
            atomicAdd(a.acc + 3 * cur_q + 2, t2);
        }
    }
}

}  // namespace

void tiles_kernel_occupancy(int* per_sm) {
    *per_sm = 0;
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(per_sm, tiles_kernel, 32 * kTileWarps, 0);
}

void launch_tiles(const SumsArgs& a, int grid, cudaStream_t s) { tiles_kernel<<<grid, 32 * kTileWarps, 0, s>>>(a); }

}  // namespace drb
