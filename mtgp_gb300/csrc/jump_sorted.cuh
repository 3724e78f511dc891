// jump_sorted.cuh -- GF(2) jump-ahead of one window by one CTA (or a share of
// it), with the taps sorted by pattern.
//
// The jumped window is the correlation (jump_device.cuh)
//
//     J[l] = XOR_{i : c_i = 1} seq[i + l],      l = 0 .. N-1,
//
// of the sequence that starts with the window.  The taps go in rows of
// eight: row a holds taps 8a .. 8a+7, its pattern p_a is byte a of the
// polynomial.  With S_p[m] = XOR_{a : p_a = p} seq[8a + m],
//
//     J[l] = XOR_b U_b[l + b],   U_b = XOR_{p : bit b of p} S_p   (b < 8),
//
// so a row costs one XOR of N + 7 words, whatever its pattern.  The rows are
// sorted by pattern in Gray-code order, in which consecutive patterns
// differ in one bit: with P the running XOR of all rows so far, U_b is the
// XOR of P taken at every change of bit b (summation by parts; the pattern
// after the last counts as 0), one more XOR per pattern.  Rows of zeros are
// left out.  Any range of the patterns can be one warp's or one CTA's share.
//
// One CTA: GW threads extend the sequence through a shared linear buffer
// (the parallel recursion, one barrier per GW words) while the other warps
// sort the rows (histogram, scan, scatter); then warp (piece, range) walks
// its range of the patterns for 128 of the words (32-bit) of the sequence
// behind the rows, four to a lane, one 128-bit shared load a row.  Polynomials longer
// than C taps go in chunks of C.
//
// Bound: shared-memory bandwidth, about 1500 rows (mexp / 8 and the padding
// of odd patterns) x 512 bytes x PIECES and a wavefront per two rows for
// their places: 21 k wavefronts a jump at MEXP 11213 plus 2 k for the
// sequence, against 27 k SM cycles a jump measured with two CTAs on every SM
// (4096 jumps in 348 us; 584 us with the unsorted taps of jump_device.cuh, a
// lone jump 18 us against 46).  Two CTAs of 80 registers beat three of 56
// (394 us: spills), and the rows of the next step loaded ahead beat loading
// them in order (383 us).
#pragma once
#include "jump_device.cuh"

namespace mtgp {

// N live words; RG row ranges per CTA; GW words per recursion step (GW <= N -
// pos for every parameter set); C taps per chunk (a multiple of 128); MINB
// CTAs per SM that fix the registers.
template <class Tr_, int N_, int RG_, int GW_, int C_, int MINB_>
struct SJump {
    using Tr = Tr_;
    using W = typename Tr::W;
    static constexpr int N = N_, RG = RG_, GW = GW_, C = C_, MINB = MINB_;
    static constexpr int WS = sizeof(W) / 4;
    static constexpr int ROW = 8 * sizeof(W);                  // bytes of one row's step
    static constexpr int PIECES = ((N + 7) * WS + 127) / 128;  // 128 32-bit words each
    static constexpr int CWARPS = PIECES * RG;
    static constexpr int GWARPS = GW / 32;
    static constexpr int WARPS = CWARPS > GWARPS + 4 ? CWARPS : GWARPS + 4;
    static constexpr int NT = 32 * WARPS;
    static constexpr int ST = NT - GW;                         // threads that sort
    // each pattern's list even, four more behind, whole warps' loops over it
    static constexpr int ROWS = (C / 8 + 260 + 31) & ~31;
    static constexpr int SEQ = C + PIECES * 128 / WS;          // words of the sequence buffer
    static constexpr int ZERO = SEQ * (int)sizeof(W);          // a row of zeros behind it
    static constexpr int NJ = (N + 3) & ~3;
    static_assert(C % 128 == 0 && GW % 32 == 0 && C >= N && C >= GW && NT <= 1024, "bad jump geometry");
    static_assert(SEQ >= C + N, "sequence buffer too small");
    // barN's conditions: its groups are whole warps, one of them at least, and
    // every loop before it runs over a multiple of 32 in steps of its group, so
    // that no two lanes of a warp leave one at different trips
    static_assert(ST % 32 == 0 && ST >= 32 && GW % 32 == 0 && ROWS % 32 == 0,
                  "a warp would reach a barrier in parts");
    static constexpr size_t off_jout = ZERO + PIECES * 512;
    static constexpr size_t off_rows = off_jout + sizeof(W) * NJ;
    static constexpr size_t off_ends = off_rows + 4 * ROWS;
    static constexpr size_t kBytes = off_ends + 4 * 256;
    static_assert(off_rows % 16 == 0, "jump buffers misaligned");
    static_assert(kBytes <= 227 * 1024, "jump buffers exceed shared memory");
};

// Barrier `id` of `threads` threads, whole warps.  The aligned form is undefined
// unless a warp's lanes arrive as one: the loops before it end at the same trip
// for all of them (SJump's static_assert), and __syncwarp brings them together
// again behind the branches inside.
__device__ __forceinline__ void barN(int id, int threads) {
    __syncwarp();
    asm volatile("barrier.sync.aligned %0, %1;" ::"r"(id), "r"(threads) : "memory");
}

// Rank of pattern p in Gray-code order (p = rank ^ rank >> 1).
__device__ __forceinline__ uint32_t grayRank(uint32_t p) {
    p ^= p >> 4;
    p ^= p >> 2;
    return p ^ (p >> 1);
}

// The pattern of this rank belongs to the share [u0, u1) of kJumpUnits.
static_assert(kJumpUnits * 8 == 256, "a unit is eight ranks");
__device__ __forceinline__ bool inShare(uint32_t rank, int u0, int u1) {
    return rank - 8u * (uint32_t)u0 < 8u * (uint32_t)(u1 - u0);
}

__device__ __forceinline__ void xor4(uint4 &a, const uint4 &b) {
    a.x ^= b.x;
    a.y ^= b.y;
    a.z ^= b.z;
    a.w ^= b.w;
}

// Word k (constant after unrolling) of the 4 of a lane.
__device__ __forceinline__ uint32_t wordOf(const uint4 &v, int k) {
    return k == 0 ? v.x : k == 1 ? v.y : k == 2 ? v.z : v.w;
}

// The jump of the window in seq[0 .. N) by pg (nwords words), its patterns
// [u0, u1) of kJumpUnits only: the result (to be XOR-ed with the other
// parts') is in jout[0 .. N) on return.  smem: SJump::kBytes bytes, seq
// first.  All NT threads call it after the window is written; it begins and
// ends with a barrier.
template <class G>
__device__ __forceinline__ void jumpSorted(unsigned char *smem, const typename G::Tr::Lane &L,
                                           const uint32_t *__restrict__ pg, int nwords, int u0,
                                           int u1) {
    using Tr = typename G::Tr;
    using W = typename G::W;
    constexpr int N = G::N, C = G::C, GW = G::GW, NT = G::NT, ST = G::ST, RG = G::RG, WS = G::WS;
    W *seq = reinterpret_cast<W *>(smem);
    W *jout = reinterpret_cast<W *>(smem + G::off_jout);
    uint32_t *rows = reinterpret_cast<uint32_t *>(smem + G::off_rows);
    uint32_t *ends = reinterpret_cast<uint32_t *>(smem + G::off_ends);
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int pc = warp % G::PIECES, rg = warp / G::PIECES;
    uint4 U[8];
#pragma unroll
    for (int b = 0; b < 8; b++) U[b] = make_uint4(0, 0, 0, 0);
    for (int k = tid; k < N; k += NT) jout[k] = 0;
    for (int k = tid; k < G::PIECES * 128; k += NT)
        reinterpret_cast<uint32_t *>(smem + G::ZERO)[k] = 0;

    for (int c0 = 0;; c0 += C) {
        __syncthreads();
        const int left = nwords * 32 - c0;
        const int taps = left < C ? left : C;
        if (tid < GW) {
            // extend the sequence to the last word that a tap reads; the last
            // step ends there, making some words of the step before again
            const int need = (taps > GW ? taps : GW) + N;
            for (int w = N; w < need; w += GW) {
                const int i = (w < need - GW ? w : need - GW) + tid;
                const W x1 = seq[i - N], x2 = seq[i - N + 1], y = seq[i - N + L.pos];
                seq[i] = Tr::rec(x1, x2, y, L);
                barN(1, GW);
            }
        } else {
            // this share's rows with taps, sorted by the rank of their pattern
            const int st = tid - GW;
            constexpr int PER = (C / 32 + ST - 1) / ST;
            uint32_t pv[PER];
#pragma unroll
            for (int i = 0; i < PER; i++) {
                const int k = st + i * ST;
                pv[i] = k < taps / 32 ? pg[c0 / 32 + k] : 0u;
            }
            for (int k = st; k < 256; k += ST) ends[k] = 0;
            for (int k = st; k < G::ROWS; k += ST) rows[k] = G::ZERO;
            barN(2, ST);
#pragma unroll
            for (int i = 0; i < PER; i++)
#pragma unroll
                for (int q = 0; q < 4; q++) {
                    const uint32_t p = (pv[i] >> (8 * q)) & 255u;
                    const uint32_t rank = grayRank(p);
                    if (p && inShare(rank, u0, u1)) atomicAdd(&ends[rank], 1u);
                }
            barN(2, ST);
            if (st < 32) {  // exclusive scan, eight bins a lane
                uint32_t h[8], sum = 0;
#pragma unroll
                for (int q = 0; q < 8; q++) {
                    h[q] = (ends[8 * lane + q] + 1) & ~1u;
                    sum += h[q];
                }
                uint32_t at = sum;
#pragma unroll
                for (int d = 1; d < 32; d <<= 1) {
                    const uint32_t v = __shfl_up_sync(kFull, at, d);
                    if (lane >= d) at += v;
                }
                at -= sum;
#pragma unroll
                for (int q = 0; q < 8; q++) {
                    ends[8 * lane + q] = at;
                    at += h[q];
                }
            }
            barN(2, ST);
#pragma unroll
            for (int i = 0; i < PER; i++)
#pragma unroll
                for (int q = 0; q < 4; q++) {
                    const uint32_t p = (pv[i] >> (8 * q)) & 255u;
                    const uint32_t rank = grayRank(p);
                    if (p && inShare(rank, u0, u1))
                        rows[atomicAdd(&ends[rank], 1u)] =
                            (uint32_t)(4 * (st + i * ST) + q) * (uint32_t)G::ROW;
                }
        }
        __syncthreads();
        if (warp < G::CWARPS) {
            const int n = u1 - u0, ua = u0 + n * rg / RG, ub = u0 + n * (rg + 1) / RG;
            const unsigned char *base = smem + pc * 512 + lane * 16;
            auto row = [base](uint32_t o) { return *reinterpret_cast<const uint4 *>(base + o); };
            // two rows a step; the next step's rows and the places of those
            // after them are on the way meanwhile (into the next patterns')
            int k = ua ? ((int)ends[8 * ua - 1] + 1) & ~1 : 0;
            uint2 o = *reinterpret_cast<const uint2 *>(rows + k);
            uint4 P = make_uint4(0, 0, 0, 0), a = row(o.x), b = row(o.y);
            o = *reinterpret_cast<const uint2 *>(rows + k + 2);
            for (int u = ua; u < ub; u++) {
                // ranks 8u .. 8u + 7: the bit that changes after each is
                // fixed but for the last
#pragma unroll
                for (int q = 0; q < 8; q++) {
                    const int end = (int)ends[8 * u + q];
#pragma unroll 1
                    for (; k < end; k += 2) {
                        P.x ^= a.x ^ b.x;
                        P.y ^= a.y ^ b.y;
                        P.z ^= a.z ^ b.z;
                        P.w ^= a.w ^ b.w;
                        a = row(o.x);
                        b = row(o.y);
                        o = *reinterpret_cast<const uint2 *>(rows + k + 4);
                    }
                    if (q < 7) xor4(U[q & 1 ? q & 2 ? 2 : 1 : 0], P);
                }
                const uint32_t r = 8u * (uint32_t)u + 7u, p = r ^ (r >> 1);
                const uint32_t d = u + 1 == ub ? p : p ^ (r + 1) ^ ((r + 1) >> 1);
#pragma unroll
                for (int b = 2; b < 8; b++)
                    if ((d >> b) & 1) xor4(U[b], P);
            }
        }
        if (c0 + C >= nwords * 32) break;
        __syncthreads();
        for (int k = tid; k < N; k += NT) seq[k] = seq[C + k];  // C >= N: no overlap
    }

    // J[l] = XOR_b U_b[l + b]: this lane's words of the sum come from it and
    // the lanes above; the first words of a piece also belong to the last
    // outputs of the piece below
    if (warp < G::CWARPS) {
        uint32_t *j32 = reinterpret_cast<uint32_t *>(jout);
        const int at = pc * 128 + 4 * lane;
        uint32_t J[4] = {0, 0, 0, 0};
#pragma unroll
        for (int b = 0; b < 8; b++)
#pragma unroll
            for (int k = 0; k < 4; k++) {
                const int up = (k + b * WS) >> 2, w = (k + b * WS) & 3;
                uint32_t v = wordOf(U[b], w);
                if (up) {
                    v = __shfl_down_sync(kFull, v, up);
                    if (lane + up > 31) v = 0;
                }
                J[k] ^= v;
            }
#pragma unroll
        for (int k = 0; k < 4; k++)
            if (at + k < N * WS) atomicXor(&j32[at + k], J[k]);
        if (pc > 0) {
#pragma unroll
            for (int b = 1; b < 8; b++)
#pragma unroll
                for (int k = 0; k < 4; k++) {
                    const int t = 4 * lane + k - b * WS;  // < 0: in the piece below
                    if (t < 0 && pc * 128 + t < N * WS) atomicXor(&j32[pc * 128 + t], wordOf(U[b], k));
                }
        }
    }
    __syncthreads();
}

}  // namespace mtgp
