// jump_kernels.cu -- jump-ahead of many windows, one team of CTAs per
// descriptor.
//
// Each descriptor names a source window, a destination window and a chain
// of polynomials (jump_sorted.cuh).  Substream j of the reference's CUDA
// sample is reached the same way, from the table of X^(4^k * 3^162) mod chi
// (cuda-sample/mtgp32-jump-kernel.cuh:383-401), but there one thread steps
// the recursion for every coefficient; here the whole CTA does.
#include "cta_team.cuh"
#include "jump_sorted.cuh"

namespace mtgp {

namespace {

// A team of CS CTAs per descriptor, each with its share of every polynomial's
// patterns; all make the sequence, which takes them as long as one.
template <class G, int CS>
__global__ void __launch_bounds__(G::NT, G::MINB)
k_jump(const typename G::Tr::P *__restrict__ params, typename G::W *__restrict__ states,
       const JumpDesc *__restrict__ descs, const __grid_constant__ JumpDesc row, int nwords) {
    using W = typename G::W;
    extern __shared__ __align__(16) unsigned char smem[];
    const Team<CS> team;
    W *seq = reinterpret_cast<W *>(smem);
    W *jout = reinterpret_cast<W *>(smem + G::off_jout);
    const JumpDesc &D = descs ? descs[blockIdx.x / CS] : row;
    const uint64_t at = descs ? 0 : blockIdx.x / CS * row.step;
    typename G::Tr::Lane L;
    L.load(params[D.pidx], threadIdx.x & 31);
    for (int k = threadIdx.x; k < G::N; k += G::NT) seq[k] = states[D.src + at + k];
    for (int c = 0; c < D.nchain; c++) {
        jumpSorted<G>(smem, L, D.poly[c], nwords, kJumpUnits * team.rank / CS,
                      kJumpUnits * (team.rank + 1) / CS);
        if constexpr (CS > 1) team.sync();
        for (int k = threadIdx.x; k < G::N; k += G::NT) seq[k] = team.sum(jout + k);
        if constexpr (CS > 1) team.sync();  // before any CTA clears its share, or ends
    }
    if (team.rank == 0)
        for (int k = threadIdx.x; k < G::N; k += G::NT) states[D.dst + at + k] = seq[k];
}

// A team of CS CTAs per jump of one window by polynomials of their own: window
// dst[D.dst] of each, polynomial D.poly (-1: a copy).
template <class G, int CS>
__global__ void __launch_bounds__(G::NT, G::MINB)
k_jump_fan(const typename G::Tr::P *__restrict__ params, const typename G::W *__restrict__ states,
           const uint32_t *__restrict__ polys, int nwords, typename G::W *__restrict__ dst,
           int stride, const JumpPart *__restrict__ parts) {
    using W = typename G::W;
    extern __shared__ __align__(16) unsigned char smem[];
    const Team<CS> team;
    W *seq = reinterpret_cast<W *>(smem);
    W *jout = reinterpret_cast<W *>(smem + G::off_jout);
    const JumpPart &D = parts[blockIdx.x / CS];
    W *to = dst + (size_t)D.dst * stride;
    if (D.poly < 0) {  // the whole team
        if (team.rank == 0)
            for (int k = threadIdx.x; k < G::N; k += G::NT) to[k] = states[D.src + k];
        return;
    }
    typename G::Tr::Lane L;
    L.load(params[D.pidx], threadIdx.x & 31);
    for (int k = threadIdx.x; k < G::N; k += G::NT) seq[k] = states[D.src + k];
    jumpSorted<G>(smem, L, polys + (size_t)D.poly * nwords, nwords, kJumpUnits * team.rank / CS,
                  kJumpUnits * (team.rank + 1) / CS);
    if constexpr (CS > 1) team.sync();
    for (int k = team.rank * G::NT + threadIdx.x; k < G::N; k += CS * G::NT) to[k] = team.sum(jout + k);
    if constexpr (CS > 1) team.sync();  // before any CTA ends
}

// One CTA per (jump, share of its rows): XOR-ed into the zeroed destination
// window.
template <class G>
__global__ void __launch_bounds__(G::NT, G::MINB)
k_jump_part(const typename G::Tr::P *__restrict__ params, const typename G::W *__restrict__ states,
            const uint32_t *__restrict__ polys, int nwords, typename G::W *__restrict__ dst,
            int stride, const JumpPart *__restrict__ parts) {
    using W = typename G::W;
    extern __shared__ __align__(16) unsigned char smem[];
    W *seq = reinterpret_cast<W *>(smem);
    const W *jout = reinterpret_cast<const W *>(smem + G::off_jout);
    const JumpPart &D = parts[blockIdx.x];
    typename G::Tr::Lane L;
    L.load(params[D.pidx], threadIdx.x & 31);
    for (int k = threadIdx.x; k < G::N; k += G::NT) seq[k] = states[D.src + k];
    jumpSorted<G>(smem, L, polys + (size_t)D.poly * nwords, nwords, D.u0, D.u1);
    W *to = dst + (size_t)D.dst * stride;
    for (int k = threadIdx.x; k < G::N; k += G::NT) G::Tr::axor(&to[k], jout[k]);
}

// The longer exponents: the taps unsorted, against a ring that holds part of
// the sequence (jump_device.cuh).  Early forms of the sorted kernel did not end
// at MEXP 44497 (704 threads).  The first had the aligned barrier, without a
// __syncwarp, behind loops that a warp's lanes left at different trips, which
// is undefined; of the second, with the unaligned barrier, the cause is not
// known.  The shapes that the sorted kernel is run with reach every barrier by
// whole warps, each lane at the same trip (SJump, barN), in loops whose bounds
// are the same for a barrier's whole group; MEXP 44497 and 110503 have not been
// run with this form.
template <class Tr, class Geo>
__global__ void __launch_bounds__(Geo::NT)
k_jump_ring(const typename Tr::P *__restrict__ params, typename Tr::W *__restrict__ states,
            const JumpDesc *__restrict__ descs, const __grid_constant__ JumpDesc row, int nwords) {
    using W = typename Tr::W;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    W *smem = reinterpret_cast<W *>(smem_raw);
    const JumpDesc &D = descs ? descs[blockIdx.x] : row;
    const uint64_t at = descs ? 0 : blockIdx.x * row.step;
    typename Tr::Lane L;
    L.load(params[D.pidx], threadIdx.x & 31);
    for (int k = threadIdx.x; k < Geo::N; k += Geo::NT) smem[k] = states[D.src + at + k];
    jump_chain<Tr, Geo>(smem, L, D.poly, D.nchain, nwords);
    for (int k = threadIdx.x; k < Geo::N; k += Geo::NT) states[D.dst + at + k] = smem[k];
}

// A share [u0, u1) of kJumpUnits here is a range of whole chunks of taps.  A
// part makes the sequence up to its last chunk, so rounding up gives the odd
// chunks to the earlier parts (11 chunks in 4 parts: 3, 3, 3, 2; with 2, 3, 3,
// 3 the parts of 76 jumps at 64-bit MEXP 44497 took 181 us instead of 170).
__host__ __device__ constexpr int ringChunk(int chunks, int unit) {
    return (chunks * unit + kJumpUnits - 1) / kJumpUnits;
}
static_assert(ringChunk(11, 0) == 0 && ringChunk(11, 8) == 3 && ringChunk(11, 24) == 9 &&
                  ringChunk(11, 32) == 11,
              "every chunk once, the odd ones to the earlier parts");
template <class Tr, class Geo>
__global__ void __launch_bounds__(Geo::NT)
k_jump_part_ring(const typename Tr::P *__restrict__ params,
                 const typename Tr::W *__restrict__ states, const uint32_t *__restrict__ polys,
                 int nwords, typename Tr::W *__restrict__ dst, int stride,
                 const JumpPart *__restrict__ parts) {
    using W = typename Tr::W;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    W *smem = reinterpret_cast<W *>(smem_raw);
    const JumpPart &D = parts[blockIdx.x];
    typename Tr::Lane L;
    L.load(params[D.pidx], threadIdx.x & 31);
    for (int k = threadIdx.x; k < Geo::N; k += Geo::NT) smem[k] = states[D.src + k];
    __syncthreads();
    const int chunks = (nwords * 32 + Geo::C - 1) / Geo::C;
    jump_part<Tr, Geo>(smem, L, polys + (size_t)D.poly * nwords, nwords,
                       ringChunk(chunks, D.u0), ringChunk(chunks, D.u1),
                       dst + (size_t)D.dst * stride);
}

template <class Tr, class Geo>
struct Ring {};  // selects the unsorted kernels

template <class Tr, class Geo>
cudaError_t launchParts(Ring<Tr, Geo>, const typename Tr::P *params, const typename Tr::W *states,
                        const uint32_t *polys, int nwords, typename Tr::W *dst, int stride,
                        const JumpPart *parts, int nparts, cudaStream_t s) {
    const size_t smem = Geo::template bytes<typename Tr::W>(nwords);
    static std::atomic<size_t> seen[16];
    cudaError_t e = allowSmem(k_jump_part_ring<Tr, Geo>, smem, seen);
    if (e != cudaSuccess) return e;
    if (nparts <= 0) return cudaSuccess;
    k_jump_part_ring<Tr, Geo><<<nparts, Geo::NT, smem, s>>>(params, states, polys, nwords, dst,
                                                            stride, parts);
    return cudaGetLastError();
}

template <class Tr, class Geo>
cudaError_t launch(Ring<Tr, Geo>, const typename Tr::P *params, typename Tr::W *states,
                   const JumpDesc *descs, int ndesc, int nwords, cudaStream_t s,
                   const JumpDesc &row) {
    const size_t smem = Geo::template bytes<typename Tr::W>(nwords);
    static std::atomic<size_t> seen[16];
    cudaError_t e = allowSmem(k_jump_ring<Tr, Geo>, smem, seen);
    if (e != cudaSuccess) return e;
    if (ndesc <= 0) return cudaSuccess;
    k_jump_ring<Tr, Geo><<<ndesc, Geo::NT, smem, s>>>(params, states, descs, row, nwords);
    return cudaGetLastError();
}

template <class G, int CS>
cudaError_t launchFanTeam(const typename G::Tr::P *params, const typename G::W *states,
                          const uint32_t *polys, int nwords, typename G::W *dst, int stride,
                          const JumpPart *jumps, int n, cudaStream_t s) {
    static std::atomic<size_t> seen[16];
    cudaError_t e = allowSmem(k_jump_fan<G, CS>, G::kBytes, seen);
    if (e != cudaSuccess) return e;
    return launchTeams(k_jump_fan<G, CS>, n, CS, G::NT, G::kBytes, s, params, states, polys,
                       nwords, dst, stride, jumps);
}

template <class G>
cudaError_t launchFan(G, const typename G::Tr::P *params, const typename G::W *states,
                      const uint32_t *polys, int nwords, typename G::W *dst, int stride,
                      const JumpPart *jumps, int n, int cs, cudaStream_t s) {
    if (n <= 0) return cudaSuccess;
    if (cs >= 8) return launchFanTeam<G, 8>(params, states, polys, nwords, dst, stride, jumps, n, s);
    if (cs >= 4) return launchFanTeam<G, 4>(params, states, polys, nwords, dst, stride, jumps, n, s);
    if (cs >= 2) return launchFanTeam<G, 2>(params, states, polys, nwords, dst, stride, jumps, n, s);
    return launchFanTeam<G, 1>(params, states, polys, nwords, dst, stride, jumps, n, s);
}

// single fills are split only where the jump kernel sorts
template <class Tr, class Geo>
cudaError_t launchFan(Ring<Tr, Geo>, const typename Tr::P *, const typename Tr::W *,
                      const uint32_t *, int, typename Tr::W *, int, const JumpPart *, int, int,
                      cudaStream_t) {
    return cudaErrorInvalidValue;
}

template <class G>
cudaError_t launchParts(G, const typename G::Tr::P *params, const typename G::W *states,
                        const uint32_t *polys, int nwords, typename G::W *dst, int stride,
                        const JumpPart *parts, int nparts, cudaStream_t s) {
    static std::atomic<size_t> seen[16];
    cudaError_t e = allowSmem(k_jump_part<G>, G::kBytes, seen);
    if (e != cudaSuccess) return e;
    if (nparts <= 0) return cudaSuccess;
    k_jump_part<G><<<nparts, G::NT, G::kBytes, s>>>(params, states, polys, nwords, dst, stride,
                                                    parts);
    return cudaGetLastError();
}

template <class G, int CS>
cudaError_t launchTeam(const typename G::Tr::P *params, typename G::W *states,
                       const JumpDesc *descs, int ndesc, int nwords, cudaStream_t s,
                       const JumpDesc &row) {
    static std::atomic<size_t> seen[16];
    cudaError_t e = allowSmem(k_jump<G, CS>, G::kBytes, seen);
    if (e != cudaSuccess) return e;
    return launchTeams(k_jump<G, CS>, ndesc, CS, G::NT, G::kBytes, s, params, states, descs, row,
                       nwords);
}

template <class G>
cudaError_t launch(G, const typename G::Tr::P *params, typename G::W *states, const JumpDesc *descs,
                   int ndesc, int nwords, cudaStream_t s, const JumpDesc &row) {
    if (ndesc <= 0) return cudaSuccess;
    switch (teamSize(ndesc, smCount())) {
    case 8: return launchTeam<G, 8>(params, states, descs, ndesc, nwords, s, row);
    case 4: return launchTeam<G, 4>(params, states, descs, ndesc, nwords, s, row);
    case 2: return launchTeam<G, 2>(params, states, descs, ndesc, nwords, s, row);
    default: return launchTeam<G, 1>(params, states, descs, ndesc, nwords, s, row);
    }
}

}  // namespace

// Per exponent: live words, row ranges per CTA, words per recursion step,
// taps per chunk, CTAs per SM.  The chunk is the whole polynomial where the
// sequence then leaves room for two or three CTAs per SM, half of it at
// MEXP 23209.
constexpr int kRingThreads = 256;
#define MTGP_JGEO32(X)                                              \
    X(11213, (SJump<Tr32, 351, 4, 256, 11264, 2>))                  \
    X(23209, (SJump<Tr32, 726, 2, 256, 11648, 2>))                  \
    X(44497, (Ring<Tr32, JGeo<1391, 45, kRingThreads, 256, 4096>>))
#define MTGP_JGEO64(X)                                              \
    X(11213, (SJump<Tr64, 176, 4, 128, 11264, 2>))                  \
    X(23209, (SJump<Tr64, 363, 2, 256, 11648, 2>))                  \
    X(44497, (Ring<Tr64, JGeo<696, 23, kRingThreads, 256, 4096>>))  \
    X(110503, (Ring<Tr64, JGeo<1727, 27, kRingThreads, 256, 4096>>))

template <class G> struct Unwrap;
template <class G> struct Unwrap<void(G)> { using T = G; };
#define UNWRAP(G) typename Unwrap<void G>::T

cudaError_t launchJump32(int mexp, const DevParams32 *params, uint32_t *states,
                         const JumpDesc *descs, int ndesc, int nwords, cudaStream_t s,
                         const JumpDesc &row) {
#define X(M, G) \
    if (mexp == M) return launch(UNWRAP(G)(), params, states, descs, ndesc, nwords, s, row);
    MTGP_JGEO32(X)
#undef X
    return cudaErrorInvalidValue;
}

cudaError_t launchJump64(int mexp, const DevParams64 *params, uint64_t *states,
                         const JumpDesc *descs, int ndesc, int nwords, cudaStream_t s,
                         const JumpDesc &row) {
#define X(M, G) \
    if (mexp == M) return launch(UNWRAP(G)(), params, states, descs, ndesc, nwords, s, row);
    MTGP_JGEO64(X)
#undef X
    return cudaErrorInvalidValue;
}

cudaError_t launchJumpParts32(int mexp, const DevParams32 *params, const uint32_t *states,
                              const uint32_t *polys, int nwords, uint32_t *dst, int stride,
                              const JumpPart *parts, int nparts, cudaStream_t s) {
#define X(M, G)                                                                              \
    if (mexp == M)                                                                          \
        return launchParts(UNWRAP(G)(), params, states, polys, nwords, dst, stride, parts, \
                                            nparts, s);
    MTGP_JGEO32(X)
#undef X
    return cudaErrorInvalidValue;
}

cudaError_t launchJumpParts64(int mexp, const DevParams64 *params, const uint64_t *states,
                              const uint32_t *polys, int nwords, uint64_t *dst, int stride,
                              const JumpPart *parts, int nparts, cudaStream_t s) {
#define X(M, G)                                                                              \
    if (mexp == M)                                                                          \
        return launchParts(UNWRAP(G)(), params, states, polys, nwords, dst, stride, parts, \
                                            nparts, s);
    MTGP_JGEO64(X)
#undef X
    return cudaErrorInvalidValue;
}

cudaError_t launchJumpFan32(int mexp, const DevParams32 *params, const uint32_t *states,
                            const uint32_t *polys, int nwords, uint32_t *dst, int stride,
                            const JumpPart *jumps, int n, int cs, cudaStream_t s) {
#define X(M, G)                                                                                 \
    if (mexp == M)                                                                             \
        return launchFan(UNWRAP(G)(), params, states, polys, nwords, dst, stride, jumps, n, cs, s);
    MTGP_JGEO32(X)
#undef X
    return cudaErrorInvalidValue;
}

cudaError_t launchJumpFan64(int mexp, const DevParams64 *params, const uint64_t *states,
                            const uint32_t *polys, int nwords, uint64_t *dst, int stride,
                            const JumpPart *jumps, int n, int cs, cudaStream_t s) {
#define X(M, G)                                                                                 \
    if (mexp == M)                                                                             \
        return launchFan(UNWRAP(G)(), params, states, polys, nwords, dst, stride, jumps, n, cs, s);
    MTGP_JGEO64(X)
#undef X
    return cudaErrorInvalidValue;
}

}  // namespace mtgp
