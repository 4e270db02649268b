// Units of a dense product with both factors' lower levels in shared memory:
// shared by the series, row-resident product and chain kernels.
#pragma once

#include <algorithm>
#include <type_traits>

#include "common.cuh"

namespace rpyb {

template <int D, int E>
struct Power {
    static constexpr int value = D * Power<D, E - 1>::value;
};
template <int D>
struct Power<D, 0> {
    static constexpr int value = 1;
};
// first word of level K
template <int D, int K>
struct LevelStart {
    static constexpr int value = LevelStart<D, K - 1>::value + Power<D, K - 1>::value;
};
template <int D>
struct LevelStart<D, 0> {
    static constexpr int value = 0;
};

// acc[u] += sum over p = K - 1 down to 1 of R_p (x) X_{K-p} at the words
// u D^(K-F) + r of level K >= F (u over the first F letters, r the others), the
// lower levels of R and X as float64 in shared memory.  Every split is
// unrolled: word offsets are immediates, and a split costs one division by D,
// two addresses and U + 1 shared loads.  Lanes of consecutive r read right
// words as conflict-free runs and left words as broadcasts or short runs.
template <int D, int F, int K, int U>
__device__ __forceinline__ void split_unit(double (&acc)[U], const double* R, const double* X,
                                            uint32_t r)
{
    // from the shortest right part up, peeling a letter a step
    uint32_t q = r, m = 0;
    auto split = [&](auto sc) {
        constexpr int s = decltype(sc)::value;
        const uint32_t q2 = q / (uint32_t)D;
        m += (q - q2 * (uint32_t)D) * (uint32_t)Power<D, s - 1>::value;
        q = q2;
        constexpr int run = Power<D, K - s - F>::value;
        const double x = X[LevelStart<D, s>::value + m];
        const double* rp = R + LevelStart<D, K - s>::value + q;
#pragma unroll
        for (int u = 0; u < U; ++u) acc[u] = fma(rp[u * run], x, acc[u]);
    };
    auto walk = [&](auto self, auto sc) {
        constexpr int s = decltype(sc)::value;
        if constexpr (s <= K - F) {
            split(sc);
            self(self, std::integral_constant<int, s + 1>{});
        }
    };
    walk(walk, std::integral_constant<int, 1>{});
    // splits inside the owned first letters, p = 2 then 1
    if constexpr (F >= 3 && K >= 3) {
        constexpr int rest = Power<D, F - 2>::value, run = Power<D, K - F>::value;
        const double* xp = X + LevelStart<D, K - 2>::value + r;
#pragma unroll
        for (int u = 0; u < U; ++u)
            acc[u] = fma(R[LevelStart<D, 2>::value + u / rest], xp[(u % rest) * run], acc[u]);
    }
    if constexpr (F >= 2 && K >= 2) {
        constexpr int rest = Power<D, F - 1>::value, run = Power<D, K - F>::value;
        const double* xp = X + LevelStart<D, K - 1>::value + r;
#pragma unroll
        for (int u = 0; u < U; ++u)
            acc[u] = fma(R[LevelStart<D, 1>::value + u / rest], xp[(u % rest) * run], acc[u]);
    }
}

// The same for a runtime width (F = 1, up to 16 words a unit).
__device__ __forceinline__ void split_unit_any(double (&acc)[16], const double* R, const double* X,
                                                const int64_t* db, const int64_t* pw,
                                                uint32_t d, int k, uint32_t r)
{
    uint32_t q = r, m = 0, ds = 1;
    for (int s = 1; s < k; ++s) {
        const uint32_t q2 = q / d;
        m += (q - q2 * d) * ds;
        q = q2;
        ds *= d;
        const int p = k - s;
        const double x = X[db[s] + m];
        const double* rp = R + db[p] + q;
        const uint32_t run = (uint32_t)pw[p - 1];
#pragma unroll
        for (int u = 0; u < 16; ++u)
            if (u < (int)d) acc[u] = fma(rp[u * run], x, acc[u]);
    }
}

// Calls f(k as a compile-time constant) for a level F <= k <= KMAX.
template <int F, int KMAX, typename Fn>
__device__ __forceinline__ void with_level(int k, Fn&& f)
{
    if constexpr (KMAX >= F) {
        if (k == KMAX) f(std::integral_constant<int, KMAX>{});
        else with_level<F, KMAX - 1>(k, f);
    }
}

// Threads of a block that has a whole row of top level `top` to itself, its
// units owning the first F letters.  An SM gets 1024 threads over the blocks it
// will hold: those that fit in its shared memory (`room` bytes) or, with fewer
// rows, its share of them.  A block has no use for more than one thread a unit
// of the top level, or of all levels where SMs are not full anyway.  (Counting
// only the blocks that fit left SMs idle below a dozen rows each: (5,5) float32
// x 148 accumulating took 15.1 us with 64 threads a row, 4.9 with 544.)
inline int64_t row_block_threads(const Geometry& g, int top, int F, size_t smem, int64_t room,
                                 int64_t rows, int64_t most)
{
    const int64_t resident =
        std::max<int64_t>(1, std::min<int64_t>({16, room / (int64_t)(smem + 1024), (rows + 147) / 148}));
    int64_t units = resident < 16 && F > 1 ? 32 : 0;   // the short levels' task
    for (int k = resident < 16 ? F : std::max(F, top); k <= top; ++k)
        units += (g.pw[k - F] + 31) / 32 * 32;
    // whole warps; eleven or twelve blocks of two warps are fewer than ten of three
    int64_t share = std::max<int64_t>(64, 1024 / resident / 32 * 32);
    if (share == 64 && 1024 / resident >= 85) share = 96;
    return std::max<int64_t>(32, std::min<int64_t>({units, share, most}));
}

// Room for n words staged by stage_words, in float64 words (16-byte multiple).
__host__ __device__ constexpr int stage_room(int n) { return (n + 3) & ~1; }

// n words of a row into shared memory as float64, at the returned place in
// `room` (16-byte aligned, stage_room(n) words).  Float64: asynchronous copies
// of 16 bytes, with a word before the first aligned piece and after the last
// where the row starts or ends between two (8-byte copies throughout kept the
// load/store queue full: mio_throttle 16.7 cycles an issue, (8,5) 173 -> 167
// us).  Float32: words, eight of a thread's in flight (16-byte loads, whose
// odd words wait for a latency of their own, were slower: (2,12) 43 -> 58 us).
template <typename T>
__device__ __forceinline__ double* stage_words(double* room, const T* src, int n, int tid, int B)
{
    if constexpr (sizeof(T) == 8) {
        const int head = (int)((reinterpret_cast<uintptr_t>(src) >> 3) & 1);
        double* dst = room + head;
        const uint32_t to = (uint32_t)__cvta_generic_to_shared(dst);
        const int pieces = (n - head) / 2;
        for (int i = tid; i < pieces; i += B)
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(to + (head + 2 * i) * 8),
                         "l"(src + head + 2 * i)
                         : "memory");
        const int odd = tid == 0 && head ? 0 : tid == 1 && head + 2 * pieces < n ? n - 1 : -1;
        if (odd >= 0)
            asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(to + odd * 8), "l"(src + odd)
                         : "memory");
        return dst;
    } else {
        constexpr int kLoads = 8;
        for (int i0 = tid; i0 < n; i0 += kLoads * B) {
            T v[kLoads];
#pragma unroll
            for (int j = 0; j < kLoads; ++j) v[j] = i0 + j * B < n ? src[i0 + j * B] : T(0);
#pragma unroll
            for (int j = 0; j < kLoads; ++j)
                if (i0 + j * B < n) room[i0 + j * B] = (double)v[j];
        }
        return room;
    }
}

}  // namespace rpyb
