// seed_kernels.cu -- the reference's integer seeding on the device
// (mtgp32_init_state, mtgp32-fast.c:119-137; mtgp64_init_state,
// mtgp64-fast.c:124-142), one thread per stream: every word of the window is
// filled from the parameter set's hidden word, then word 0 takes the seed
// and each later word mixes in its predecessor.  A thread's 351 (or 176)
// words form one sequential chain; streams are independent, so thousands of
// streams are seeded in one launch of a few microseconds.
#include "internal.h"

namespace mtgp {
namespace {

template <typename W> struct SeedMix;
template <> struct SeedMix<uint32_t> {
    static constexpr uint32_t mul = 1812433253u;
    static constexpr int shr = 30;
    static constexpr uint32_t bytes = 0x01010101u;
    static __device__ uint32_t top(uint32_t h) { return h; }
};
template <> struct SeedMix<uint64_t> {
    static constexpr uint64_t mul = 6364136223846793005ULL;
    static constexpr int shr = 62;
    static constexpr uint64_t bytes = 0x0101010101010101ULL;
    static __device__ uint64_t top(uint64_t h) { return h >> 32; }
};

// seeds null: every stream from `one`.  A warp per CTA, so that a few thousand
// streams use all SMs; the words go to memory 32 streams x 32 words at a time,
// turned round in shared memory: a lane's own words are a stride apart, and
// storing them as they are made (OWN) takes 45 us for 4096 streams, 8.6 us this
// way.  Bound by the chain of words: a tile's rows are loaded and stored eight
// at a time around the next tile's chain, behind its latency (in a loop of
// their own after each tile 11.6 us).  Up to kOwnStreams streams OWN has fewer
// instructions beside the chain: 16 streams of MEXP 110503, 64-bit, 34 us
// against 38; 33 streams of it 42 against 40, of MEXP 44497, 32-bit, 21
// against 14.
constexpr int kOwnStreams = 16;
template <typename W, class P, bool OWN>
__global__ void __launch_bounds__(32)
k_seed(const P *__restrict__ params, const int *__restrict__ pidx, const W *__restrict__ seeds,
       W one, W *__restrict__ states, int count, int size, int stride) {
    using M = SeedMix<W>;
    __shared__ W tile[2][32][33];
    const int lane = threadIdx.x, base = blockIdx.x * 32;
    const int rows = count - base < 32 ? count - base : 32;
    const int i = base + (lane < rows ? lane : rows - 1);
    const P &p = params[pidx[i]];
    const W hidden = p.tbl[4] ^ (p.tbl[8] << 16);
    W b = M::top(hidden);
    b += b >> 16;
    b += b >> 8;
    const W fill = (b & 0xffu) * M::bytes;
    W prev = seeds ? seeds[i] : one;
    auto next = [&prev](W mix, uint32_t k) { prev = mix ^ (M::mul * (prev ^ (prev >> M::shr)) + k); };
    if constexpr (OWN) {
        if (lane >= rows) return;
        W *a = states + (size_t)i * stride;
        a[0] = prev;
        next(hidden, 1);
        a[1] = prev;
        for (int k = 2; k < size; k++) {
            next(fill, (uint32_t)k);
            a[k] = prev;
        }
        return;
    }
    tile[0][0][lane] = prev;
    next(hidden, 1);
    tile[0][1][lane] = prev;
    for (int j = 2; j < 32; j++) {
        next(fill, (uint32_t)j);
        tile[0][j][lane] = prev;
    }
    // tile k0 / 32 while the one before it is stored, and a round for the last
    for (int k0 = 32; k0 < size + 32; k0 += 32) {
        __syncwarp();
        W(*to)[33] = tile[(k0 >> 5) & 1];
        const W *from = tile[((k0 >> 5) & 1) ^ 1][lane];
        const int k = k0 - 32 + lane;
        W *out = states + (size_t)base * stride + k;
        for (int j0 = 0; j0 < 32; j0 += 8) {
            W done[8];
#pragma unroll
            for (int q = 0; q < 8; q++) done[q] = from[j0 + q];
#pragma unroll
            for (int q = 0; q < 8; q++) {
                next(fill, (uint32_t)(k0 + j0 + q));
                to[j0 + q][lane] = prev;
            }
#pragma unroll
            for (int q = 0; q < 8; q++)
                if (j0 + q < rows && k < size) out[(size_t)(j0 + q) * stride] = done[q];
        }
    }
}

// Key schedules (mtgp32_init_by_array, mtgp32-fast.c:151-235, and
// init_by_str, :250-334; 64-bit twins mtgp64-fast.c:156-239 / 255-339), one
// thread per stream.  keys[koff[i] .. koff[i+1]) are stream i's key words as
// the reference adds them (array words, or string bytes as signed char); the
// window is filled like the integer seeding's, then three passes mix keys
// and positions in.  The passes read and write four positions of the
// thread's own window per step (a dependent chain); the window lives in the
// stream's state row, cached by L1.
template <typename W> struct KeyMix;
template <> struct KeyMix<uint32_t> {
    static constexpr uint32_t mul1 = 1664525u, mul2 = 1566083941u;
    static constexpr int shr = 27;
};
template <> struct KeyMix<uint64_t> {
    static constexpr uint64_t mul1 = 2173292883993ULL, mul2 = 58885565329898161ULL;
    static constexpr int shr = 59;
};

template <typename W, class P>
__global__ void k_keyed(const P *__restrict__ params, const int *__restrict__ pidx,
                        const W *__restrict__ keys, const uint64_t *__restrict__ koff,
                        W *__restrict__ states, int count, int size, int stride) {
    using M = SeedMix<W>;
    using K = KeyMix<W>;
    const int s = blockIdx.x * blockDim.x + threadIdx.x;
    if (s >= count) return;
    const P &p = params[pidx[s]];
    const W hidden = p.tbl[4] ^ (p.tbl[8] << 16);
    W b = M::top(hidden);
    b += b >> 16;
    b += b >> 8;
    const W fill = (b & 0xffu) * M::bytes;
    W *a = states + (size_t)s * stride;
    for (int k = 1; k < size; k++) a[k] = fill;
    a[0] = hidden;
    const int lag = size >= 623 ? 11 : size >= 68 ? 7 : size >= 39 ? 5 : 3;
    const int mid = (size - lag) / 2;
    const W *key = keys + koff[s];
    const int len = (int)(koff[s + 1] - koff[s]);
    auto f1 = [](W x) { return (W)((x ^ (x >> K::shr)) * K::mul1); };
    auto f2 = [](W x) { return (W)((x ^ (x >> K::shr)) * K::mul2); };
    const int total = (len + 1 > size ? len + 1 : size) - 1;
    W r = f1(a[0] ^ a[mid] ^ a[size - 1]);
    a[mid] += r;
    r += (W)len;
    a[(mid + lag) % size] += r;
    a[0] = r;
    // i runs 1, 2, ..., size - 1, 0, 1, ...; the other positions follow it
    int i = 1, im = (1 + mid) % size, iml = (1 + mid + lag) % size, ip = 0;
    auto next = [&]() {
        ip = i;
        i = i + 1 == size ? 0 : i + 1;
        im = im + 1 == size ? 0 : im + 1;
        iml = iml + 1 == size ? 0 : iml + 1;
    };
    for (int j = 0; j < total; j++) {
        W t = f1(a[i] ^ a[im] ^ a[ip]);
        a[im] += t;
        t += (j < len ? key[j] : (W)0) + (W)i;
        a[iml] += t;
        a[i] = t;
        next();
    }
    for (int j = 0; j < size; j++) {
        W t = f2(a[i] + a[im] + a[ip]);
        a[im] ^= t;
        t -= (W)i;
        a[iml] ^= t;
        a[i] = t;
        next();
    }
    if (a[size - 1] == 0) a[size - 1] = (W)0x4d544750u;
}

}  // namespace

cudaError_t launchKeyed32(const DevParams32 *params, const int *pidx, const uint32_t *keys,
                          const uint64_t *koff, uint32_t *states, int count, int size, int stride,
                          cudaStream_t s) {
    if (count <= 0) return cudaSuccess;
    k_keyed<uint32_t, DevParams32><<<(count + 63) / 64, 64, 0, s>>>(params, pidx, keys, koff,
                                                                    states, count, size, stride);
    return cudaGetLastError();
}

cudaError_t launchKeyed64(const DevParams64 *params, const int *pidx, const uint64_t *keys,
                          const uint64_t *koff, uint64_t *states, int count, int size, int stride,
                          cudaStream_t s) {
    if (count <= 0) return cudaSuccess;
    k_keyed<uint64_t, DevParams64><<<(count + 63) / 64, 64, 0, s>>>(params, pidx, keys, koff,
                                                                    states, count, size, stride);
    return cudaGetLastError();
}

cudaError_t launchSeed32(const DevParams32 *params, const int *pidx, const uint32_t *seeds, uint32_t one,
                         uint32_t *states, int count, int size, int stride, cudaStream_t s) {
    if (count <= 0) return cudaSuccess;
    auto kern = count <= kOwnStreams ? k_seed<uint32_t, DevParams32, true>
                                     : k_seed<uint32_t, DevParams32, false>;
    kern<<<(count + 31) / 32, 32, 0, s>>>(params, pidx, seeds, one, states, count, size, stride);
    return cudaGetLastError();
}

cudaError_t launchSeed64(const DevParams64 *params, const int *pidx, const uint64_t *seeds, uint64_t one,
                         uint64_t *states, int count, int size, int stride, cudaStream_t s) {
    if (count <= 0) return cudaSuccess;
    auto kern = count <= kOwnStreams ? k_seed<uint64_t, DevParams64, true>
                                     : k_seed<uint64_t, DevParams64, false>;
    kern<<<(count + 31) / 32, 32, 0, s>>>(params, pidx, seeds, one, states, count, size, stride);
    return cudaGetLastError();
}

}  // namespace mtgp
