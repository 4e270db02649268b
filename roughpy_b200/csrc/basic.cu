// Memory-bound companions of the product kernel: antipode, adjoint of left
// multiplication, and batched sparse (CSR) linear maps for Lie <-> tensor.
#include <algorithm>
#include <cstring>
#include <type_traits>

#include "common.cuh"

namespace rpyb {
namespace {

struct LevelTab {
    int64_t db[kMaxDepth + 2];
    int64_t pw[kMaxDepth + 1];
    int depth;
    int width;
};

__device__ __forceinline__ int level_of(const LevelTab& t, int64_t i)
{
    int k = 0;
    while (k < t.depth && i >= t.db[k + 1]) ++k;
    return k;
}

// Antipode: out[w] = (-1)^k arg[rev(w)] per level (free_tensor_antipode.hpp:56-99).
// Reversing a word turns its last letters into its first, so a warp's
// consecutive words of out lie d^(k-1) apart in arg.  Levels of at least 2 L
// letters go through square tiles in shared memory: for one middle part, the
// d^L runs of d^L words (P, rev m, Q) of arg are read as runs and the runs
// (p, m, q) of out written as runs.  Lower levels, a few hundred words, are
// gathered from L1 one by one, with divisions by a compile-time width.  Before,
// every word was gathered so, with 64-bit divisions by a runtime width.
// Measured on B200, before -> after: (8,5) float32 x 1000 419 -> 76 us (3.9
// TB/s), (4,6) float64 x 3000 222 -> 73 us, (2,14) float32 x 500 393 -> 60 us,
// (2,5) float32 x 100000 90 -> 39 us (index arithmetic).

// the first `words` words of every row, one a thread (32-bit indices: the grid's
// stride past the last word fits)
template <typename T, int D, typename Index>
__global__ void antipode_words_kernel(T* out, const T* arg, int64_t ld_out, int64_t ld_arg,
                                      int64_t batch, Index words, const LevelTab t)
{
    const Index total = (Index)batch * words;
    for (Index g = blockIdx.x * (Index)blockDim.x + threadIdx.x; g < total;
         g += (Index)gridDim.x * blockDim.x) {
        const Index b = g / words;
        const uint32_t i = (uint32_t)(g - b * words);
        const int k = level_of(t, i);
        const uint32_t d = D > 0 ? (uint32_t)D : (uint32_t)t.width;
        uint32_t j = i - (uint32_t)t.db[k], rev = 0;
        for (int q = 0; q < k; ++q) {
            const uint32_t next = j / d;
            rev = rev * d + (j - next * d);
            j = next;
        }
        const T v = __ldg(arg + (int64_t)b * ld_arg + t.db[k] + rev);
        out[(int64_t)b * ld_out + i] = (k & 1) ? -v : v;
    }
}

template <int D, int L>
struct Letters {
    static constexpr int count = D * Letters<D, L - 1>::count;
    // the L digits of v in reverse
    static __device__ __forceinline__ int reverse(int v)
    {
        return (v % D) * Letters<D, L - 1>::count + Letters<D, L - 1>::reverse(v / D);
    }
};
template <int D>
struct Letters<D, 0> {
    static constexpr int count = 1;
    static __device__ __forceinline__ int reverse(int) { return 0; }
};

constexpr int kAntipodeThreads = 256;
// Words of a batch from which its upper levels go through tiles, a launch of
// their own: below, that costs more than gathering (in 32-bit arithmetic) does.
constexpr int64_t kAntipodeTiled = int64_t(1) << 19;

// levels 2 L and above: one tile a block
template <typename T, int D, int L>
__global__ void __launch_bounds__(kAntipodeThreads)
antipode_tiles_kernel(T* out, const T* arg, int64_t ld_out, int64_t ld_arg, int64_t batch,
                      uint32_t row_tiles, const LevelTab t)
{
    constexpr int S = Letters<D, L>::count;
    __shared__ T tile[S][S + 1];
    const int64_t total = batch * row_tiles;
    for (int64_t g = blockIdx.x; g < total; g += gridDim.x) {
        const int64_t b = g / row_tiles;
        uint32_t m = (uint32_t)(g - b * row_tiles);
        int k = 2 * L;
        while (m >= (uint32_t)t.pw[k - 2 * L]) m -= (uint32_t)t.pw[k++ - 2 * L];
        uint32_t rev = 0, j = m;
        for (int q = 0; q < k - 2 * L; ++q) {
            rev = rev * D + j % D;
            j /= D;
        }
        const uint32_t stride = (uint32_t)t.pw[k - L];   // between the runs of a tile
        const T* src = arg + b * ld_arg + t.db[k] + rev * (uint32_t)S;
        T* dst = out + b * ld_out + t.db[k] + m * (uint32_t)S;
        for (int e = threadIdx.x; e < S * S; e += kAntipodeThreads)
            tile[e / S][e % S] = __ldg(src + (uint32_t)(e / S) * stride + e % S);
        __syncthreads();
        for (int e = threadIdx.x; e < S * S; e += kAntipodeThreads) {
            const int p = e / S, q = e % S;
            const T v = tile[Letters<D, L>::reverse(q)][Letters<D, L>::reverse(p)];
            dst[(uint32_t)p * stride + q] = (k & 1) ? -v : v;
        }
        __syncthreads();
    }
}

// Adjoint of left multiplication (free_tensor_adjoint_left_mul.hpp:43-75):
//   out_k[i] += sum_q sum_{j < d^q} op_q[j] * arg_{k+q}[j d^k + i].
// Level starts satisfy db[k+q] = db[k] + d^k db[q], so with e = db[q] + j (the
// word's place in op) this is, for every output level k,
//   out_k[i] += sum_{e < E_k} op[e] * arg[db[k] + d^k e + i],
// one matrix-vector product with the tail of arg seen as an E_k x d^k matrix.
// Every level costs about T multiply-adds.  A level is cut into tiles of up to
// THREADS columns; the THREADS threads (a block's, or one warp's) of a tile
// are its columns times THREADS / columns slices of e, which read op as
// broadcasts or runs and arg as runs, and add their slices by a tree.  Sums
// are float64 for both element types.
//
// Four forms.  Rows of at most 64 words in large batches are a thread's a
// word.  Rows of at most 1024 words are a warp's, all tiles in turn
// (one tile a warp where there are few rows).  Longer rows that fit in shared
// memory are a block's: staged once, read once per level.  Others take a block
// per tile and re-read the row from L2.  The layout before, one thread per
// output word, left level 0, the sum over the whole row, to one thread.
// Measured on B200 with the zero fill of the result, before -> after:
// (3,7) float64, 500 rows 285 -> 36 us (the call's host time); (8,6) float64, one
// row 22 ms -> 40 us; (8,6) float32, 100 rows 27.6 ms -> 0.63 ms, bound by its
// seven reads of the rows from L2; (2,5) float32, 60000 rows 127 -> 107 us.
struct AdjointArgs {
    int64_t E[kMaxDepth + 1];        // terms per output word of level k
    int64_t db[kMaxDepth + 2];
    int64_t pw[kMaxDepth + 1];
    int32_t tile0[kMaxDepth + 2];    // first column tile of level k among a row's tiles
    int64_t ld_out, ld_op, ld_arg, batch;
    int64_t op_words, arg_words;     // words read of each row (staged form)
    int out_max;
    bool accumulate;                 // out += (else out =)
    int tiles_per_task;
    int heavy;                       // tiles of more than 64 terms a word (the lowest levels')
};

// One tile of one row by THREADS threads, t the thread's number among them.
template <typename T, int THREADS>
__device__ __forceinline__ void adjoint_tile(const AdjointArgs& a, T* __restrict__ out,
                                             const T* __restrict__ op, const T* __restrict__ arg,
                                             int tile, int t, double* part)
{
    int k = 0;
    while (tile >= a.tile0[k + 1]) ++k;
    const int n = (int)a.pw[k];
    const int c0 = (tile - a.tile0[k]) * THREADS;
    const int cols = min(THREADS, n - c0);
    int slices = 1, slice = 0;
    if (cols < THREADS) {
        slices = THREADS / cols;
        slice = t / cols;
    }
    const int i = c0 + (t - slice * cols);
    const T* ar = arg + a.db[k] + i;
    // unsigned: e passes E, which may be close to 2^31, by up to 8 slices
    const unsigned E = (unsigned)a.E[k];
    double s0 = 0.0, s1 = 0.0, s2 = 0.0, s3 = 0.0;
    if (slice < slices) {
        unsigned e = (unsigned)slice;
        for (; e + 7u * slices < E; e += 8u * slices) {
            double o[8], x[8];
#pragma unroll
            for (int u = 0; u < 8; ++u) {
                o[u] = (double)op[e + u * slices];
                x[u] = (double)ar[(int64_t)(e + u * slices) * n];
            }
            s0 = fma(o[0], x[0], fma(o[4], x[4], s0));
            s1 = fma(o[1], x[1], fma(o[5], x[5], s1));
            s2 = fma(o[2], x[2], fma(o[6], x[6], s2));
            s3 = fma(o[3], x[3], fma(o[7], x[7], s3));
        }
        for (; e < E; e += (unsigned)slices) s0 = fma((double)op[e], (double)ar[(int64_t)e * n], s0);
    }
    double sum = (s0 + s1) + (s2 + s3);
    // the slices, halved until one is left
    if constexpr (THREADS == 32) {
        for (int left = slices; left > 1;) {
            const int h = (left + 1) >> 1;
            const double other = __shfl_down_sync(0xffffffffu, sum, h * cols);
            if (slice + h < left) sum += other;
            left = h;
        }
    } else if (slices > 1) {
        part[t] = sum;
        for (int left = slices; left > 1;) {
            const int h = (left + 1) >> 1;
            __syncthreads();
            if (slice + h < left) part[t] = sum = sum + part[t + h * cols];
            left = h;
        }
        __syncthreads();   // part is free for the next tile
    }
    if (slice == 0) {
        T* o = out + a.db[k] + i;
        if (!a.accumulate) *o = (T)sum;
        else if (E > 0) *o = (T)((double)*o + sum);
    }
}

// Rows of at most 64 words in batches that fill the GPU: a thread per output
// word, its terms in turn.  A warp a row would spend a tile, with most lanes
// idle, on each level: (2,2) float64 x 30000 28.7 -> 3.6 us, (3,3) x 100000 119
// -> 78, (2,5) x 100000 187 -> 134.
constexpr int64_t kAdjointWords = 64;

template <typename T>
__global__ void __launch_bounds__(256)
adjoint_words_kernel(T* out, const T* op, const T* arg, const AdjointArgs a)
{
    const uint32_t size = (uint32_t)a.db[a.out_max + 1];
    const uint32_t total = (uint32_t)a.batch * size;
    for (uint32_t g = blockIdx.x * 256u + threadIdx.x; g < total; g += gridDim.x * 256u) {
        const uint32_t b = g / size, w = g - b * size;
        int k = 0;
        while (w >= (uint32_t)a.db[k + 1]) ++k;
        const int E = (int)a.E[k], n = (int)a.pw[k];
        const T* o = op + b * a.ld_op;
        const T* x = arg + b * a.ld_arg + w;   // word w - db[k] of level k, and on
        double sum = 0.0;
#pragma unroll 4
        for (int e = 0; e < E; ++e)
            sum = fma((double)__ldg(o + e), (double)__ldg(x + e * n), sum);
        T* y = out + b * a.ld_out + w;
        if (!a.accumulate) *y = (T)sum;
        else if (E > 0) *y = (T)((double)*y + sum);
    }
}

// a warp per task of tiles_per_task tiles of a row
template <typename T>
__global__ void __launch_bounds__(256)
adjoint_warp_kernel(T* out, const T* op, const T* arg, const AdjointArgs a)
{
    const int lane = (int)(threadIdx.x & 31);
    const uint32_t tiles = (uint32_t)a.tile0[a.out_max + 1];
    const uint32_t per_row = (tiles + a.tiles_per_task - 1) / a.tiles_per_task;
    const int64_t tasks = a.batch * per_row;
    for (int64_t task = blockIdx.x * (int64_t)(blockDim.x >> 5) + (threadIdx.x >> 5); task < tasks;
         task += (int64_t)gridDim.x * (blockDim.x >> 5)) {
        const int64_t b = per_row == 1 ? task : task / per_row;
        const int t0 = (int)(task - b * per_row) * a.tiles_per_task;
        const int t1 = min(t0 + a.tiles_per_task, (int)tiles);
        for (int tile = t0; tile < t1; ++tile)
            adjoint_tile<T, 32>(a, out + b * a.ld_out, op + b * a.ld_op, arg + b * a.ld_arg, tile,
                                lane, nullptr);
    }
}

// STAGED: a block per row, the row in shared memory; else a block per tile, or
// per group of tiles of few terms (a block of one multiply-add a thread costs
// more to start than to run)
constexpr int kAdjointGroup = 8;
constexpr int64_t kAdjointSmem = 108 * 1024;   // staged words of a block
template <typename T, int THREADS, bool STAGED>
__global__ void __launch_bounds__(THREADS)
adjoint_block_kernel(T* out, const T* op, const T* arg, const AdjointArgs a)
{
    __shared__ double part[THREADS];
    extern __shared__ __align__(16) unsigned char adjoint_smem[];
    const int t = (int)threadIdx.x;
    const int tiles = a.tile0[a.out_max + 1];
    if constexpr (STAGED) {
        T* sop = reinterpret_cast<T*>(adjoint_smem);
        T* sarg = sop + a.op_words;
        for (int64_t b = blockIdx.x; b < a.batch; b += gridDim.x) {
            const T* gop = op + b * a.ld_op;
            const T* garg = arg + b * a.ld_arg;
            __syncthreads();   // the previous row's reads are done
            constexpr int kLoads = 8;
            for (int i0 = t; i0 < (int)a.arg_words; i0 += kLoads * THREADS) {
                T v[kLoads], w[kLoads];
#pragma unroll
                for (int j = 0; j < kLoads; ++j) {
                    const int i = i0 + j * THREADS;
                    v[j] = i < (int)a.arg_words ? __ldg(garg + i) : T(0);
                    w[j] = i < (int)a.op_words ? __ldg(gop + i) : T(0);
                }
#pragma unroll
                for (int j = 0; j < kLoads; ++j) {
                    const int i = i0 + j * THREADS;
                    if (i < (int)a.arg_words) sarg[i] = v[j];
                    if (i < (int)a.op_words) sop[i] = w[j];
                }
            }
            __syncthreads();
            for (int tile = 0; tile < tiles; ++tile)
                adjoint_tile<T, THREADS>(a, out + b * a.ld_out, sop, sarg, tile, t, part);
        }
    } else {
        // tiles of many terms one a block, the others kGroup a block
        const int tasks = a.heavy + (tiles - a.heavy + kAdjointGroup - 1) / kAdjointGroup;
        const int64_t b = blockIdx.x / (unsigned)tasks;
        const int task = (int)(blockIdx.x - (unsigned)b * (unsigned)tasks);
        const int t0 = task < a.heavy ? task : a.heavy + (task - a.heavy) * kAdjointGroup;
        const int t1 = task < a.heavy ? task + 1 : min(t0 + kAdjointGroup, tiles);
        for (int tile = t0; tile < t1; ++tile)
            adjoint_tile<T, THREADS>(a, out + b * a.ld_out, op + b * a.ld_op, arg + b * a.ld_arg,
                                     tile, t, part);
    }
}

// y[b][r] += scale * sum_k val[k] * x[b][idx[k]]  (CSR), float64 accumulation;
// column indices outside [0, n_cols) are skipped.
template <typename T>
__global__ void csr_map_kernel(int64_t n_rows, int64_t n_cols, int64_t batch,
                               const int64_t* __restrict__ ptr,
                               const int64_t* __restrict__ idx, const double* __restrict__ val,
                               T* y, const T* x, int64_t ld_y, int64_t ld_x, double scale)
{
    const int64_t total = n_rows * batch;
    for (int64_t g = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; g < total;
         g += (int64_t)gridDim.x * blockDim.x) {
        const int64_t b = g / n_rows;
        const int64_t r = g - b * n_rows;
        const T* xr = x + b * ld_x;
        double acc = 0.0;
        for (int64_t k = __ldg(ptr + r), e = __ldg(ptr + r + 1); k < e; ++k) {
            const int64_t c = __ldg(idx + k);
            if ((uint64_t)c < (uint64_t)n_cols) acc = fma(__ldg(val + k), (double)__ldg(xr + c), acc);
        }
        T* yp = y + b * ld_y + r;
        *yp = (T)((double)*yp + scale * acc);
    }
}

LevelTab make_tab(const Geometry& g)
{
    LevelTab t{};
    for (int k = 0; k <= kMaxDepth + 1; ++k) t.db[k] = g.db[k];
    for (int k = 0; k <= kMaxDepth; ++k) t.pw[k] = g.pw[k];
    t.depth = g.depth;
    t.width = g.width;
    return t;
}

unsigned grid_for(int64_t total, int threads)
{
    const int64_t b = (total + threads - 1) / threads;
    return (unsigned)std::max<int64_t>(1, std::min<int64_t>(b, 148 * 64));
}

}  // namespace
}  // namespace rpyb

using namespace rpyb;

extern "C" {

RPYB_API int rpyb_ft_antipode(int dtype, int32_t width, int32_t depth, int64_t batch, void* out,
                              const void* arg, int64_t ld_out, int64_t ld_arg, void* stream)
{
    int rc;
    if (dtype != RPYB_F32 && dtype != RPYB_F64) return fail(RPYB_E_INVALID, "unsupported dtype");
    Geometry g;
    if ((rc = make_geometry(width, depth, g))) return rc;
    if (batch < 0) return fail(RPYB_E_INVALID, "negative batch");
    if (batch == 0) return RPYB_OK;
    if (!out || !arg) return fail(RPYB_E_INVALID, "null tensor pointer");
    if (batch > 1 && (ld_out < g.size() || ld_arg < g.size()))
        return fail(RPYB_E_INVALID, "row stride smaller than the tensor size");
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    const LevelTab t = make_tab(g);
    auto go = [&](auto kind, auto width, auto letters) {
        using V = decltype(kind);
        constexpr int D = decltype(width)::value, L = decltype(letters)::value;
        V* o = static_cast<V*>(out);
        const V* x = static_cast<const V*>(arg);
        int64_t words = g.size();
        if constexpr (L > 0) {
            if (depth >= 2 * L && batch * words >= kAntipodeTiled) {
                words = g.db[2 * L];
                const int64_t tiles = g.db[depth - 2 * L + 1];   // sum of d^(k - 2 L)
                const unsigned blocks = (unsigned)std::min<int64_t>(batch * tiles, 148 * 4096);
                antipode_tiles_kernel<V, D, L><<<blocks, kAntipodeThreads, 0, s>>>(
                    o, x, ld_out, ld_arg, batch, (uint32_t)tiles, t);
            }
        }
        const unsigned blocks = grid_for(words * batch, 256);
        if (words * batch < (int64_t(1) << 31))
            antipode_words_kernel<V, D, uint32_t><<<blocks, 256, 0, s>>>(o, x, ld_out, ld_arg, batch,
                                                                         (uint32_t)words, t);
        else
            antipode_words_kernel<V, D, int64_t><<<blocks, 256, 0, s>>>(o, x, ld_out, ld_arg, batch,
                                                                        words, t);
    };
    // L letters make runs of 25 to 64 words
    auto by_width = [&](auto kind) {
        switch (width) {
            case 2: go(kind, std::integral_constant<int, 2>{}, std::integral_constant<int, 5>{}); break;
            case 3: go(kind, std::integral_constant<int, 3>{}, std::integral_constant<int, 3>{}); break;
            case 4: go(kind, std::integral_constant<int, 4>{}, std::integral_constant<int, 3>{}); break;
            case 5: go(kind, std::integral_constant<int, 5>{}, std::integral_constant<int, 2>{}); break;
            case 6: go(kind, std::integral_constant<int, 6>{}, std::integral_constant<int, 2>{}); break;
            case 7: go(kind, std::integral_constant<int, 7>{}, std::integral_constant<int, 2>{}); break;
            case 8: go(kind, std::integral_constant<int, 8>{}, std::integral_constant<int, 2>{}); break;
            default: go(kind, std::integral_constant<int, 0>{}, std::integral_constant<int, 0>{}); break;
        }
    };
    if (dtype == RPYB_F64) by_width(double{});
    else by_width(float{});
    RPYB_CUDA(cudaGetLastError());
    return RPYB_OK;
}

static int adjoint_left_mul(int dtype, int32_t width, int32_t depth, int64_t batch, void* out,
                            const void* op, const void* arg, int64_t ld_out, int64_t ld_op,
                            int64_t ld_arg, const int32_t* deg, bool accumulate, void* stream)
{
    int rc;
    if (dtype != RPYB_F32 && dtype != RPYB_F64) return fail(RPYB_E_INVALID, "unsupported dtype");
    Geometry g;
    if ((rc = make_geometry(width, depth, g))) return rc;
    if (batch < 0) return fail(RPYB_E_INVALID, "negative batch");
    if (batch == 0) return RPYB_OK;
    if (!out || !op || !arg) return fail(RPYB_E_INVALID, "null tensor pointer");
    if (batch > 1 && (ld_out < g.size() || ld_op < g.size() || ld_arg < g.size()))
        return fail(RPYB_E_INVALID, "row stride smaller than the tensor size");
    int32_t b[3] = {-1, -1, -1};
    if (deg) std::memcpy(b, deg, sizeof(b));
    const int out_max = clamp_max_degree(b[0], depth);
    const int op_max = clamp_max_degree(b[1], depth);
    const int arg_max = clamp_max_degree(b[2], depth);
    // free_tensor_adjoint_left_mul.hpp:43-44 with all min degrees 0
    const int arg_hi = std::min(arg_max - 0, out_max);
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    AdjointArgs a{};
    for (int k = 0; k <= kMaxDepth + 1; ++k) a.db[k] = g.db[k];
    for (int k = 0; k <= kMaxDepth; ++k) a.pw[k] = g.pw[k];
    for (int k = 0; k <= out_max; ++k)
        a.E[k] = k <= arg_hi ? g.db[std::min(op_max, arg_hi - k) + 1] : 0;
    a.ld_out = ld_out;
    a.ld_op = ld_op;
    a.ld_arg = ld_arg;
    a.out_max = out_max;
    a.accumulate = accumulate;
    a.batch = batch;
    // op's words up to its highest degree used (never more than arg's), arg's
    // up to arg_hi
    a.arg_words = g.db[arg_hi + 1];
    a.op_words = g.db[std::min(op_max, arg_hi) + 1];
    const size_t staged = (size_t)(a.op_words + a.arg_words) * (dtype == RPYB_F64 ? 8 : 4);
    // Staged rows leave room for two blocks an SM; one block of a few long
    // rows would leave the chip idle, so there the tiles are spread over it.
    const int64_t T = g.db[out_max + 1];
    // (and the shortest rows at any batch)
    const bool words = T <= kAdjointWords && (batch >= 148 * 8 || T <= 8) &&
                       batch * T < (int64_t(1) << 31);
    const bool warp = T <= 1024;
    const bool stage = !warp && staged <= kAdjointSmem && batch >= 64;
    // columns of a tile: the threads of the kernel that is launched below
    const int threads = warp ? 32 : !stage && T >= 16384 && batch <= 64 ? 1024 : 256;
    int32_t tiles = 0;
    for (int k = 0; k <= out_max; ++k) {
        a.tile0[k] = tiles;
        tiles += (int32_t)((g.pw[k] + threads - 1) / threads);
    }
    for (int k = out_max + 1; k <= kMaxDepth + 1; ++k) a.tile0[k] = tiles;
    // a whole row a warp once the rows alone give every SM eight warps
    a.tiles_per_task = warp && batch >= 148 * 8 ? tiles : 1;
    a.heavy = 0;
    for (int k = 0; k <= out_max && a.E[k] > 64; ++k) a.heavy = a.tile0[k + 1];
    int64_t blocks = batch * (a.heavy + (tiles - a.heavy + kAdjointGroup - 1) / kAdjointGroup);
    if (warp) blocks = std::min<int64_t>((batch * (tiles / a.tiles_per_task) + 7) / 8, 148 * 64);
    else if (stage) blocks = std::min<int64_t>(batch, 1 << 20);
    if (words) blocks = grid_for(batch * T, 256);
    if (blocks > 0x7fffffff) return fail(RPYB_E_UNSUPPORTED, "batch too large");
    auto go = [&](auto kind) -> int {
        using V = decltype(kind);
        V* o = static_cast<V*>(out);
        const V* p = static_cast<const V*>(op);
        const V* x = static_cast<const V*>(arg);
        const unsigned nb = (unsigned)blocks;
        if (words) {
            adjoint_words_kernel<V><<<nb, 256, 0, s>>>(o, p, x, a);
        } else if (warp) {
            adjoint_warp_kernel<V><<<nb, 256, 0, s>>>(o, p, x, a);
        } else if (stage) {
            auto fn = adjoint_block_kernel<V, 256, true>;
            if (int rc = allow_shared_memory(fn, staged, kAdjointSmem)) return rc;
            fn<<<nb, 256, staged, s>>>(o, p, x, a);
        } else if (threads == 256) {
            adjoint_block_kernel<V, 256, false><<<nb, 256, 0, s>>>(o, p, x, a);
        } else {
            adjoint_block_kernel<V, 1024, false><<<nb, 1024, 0, s>>>(o, p, x, a);
        }
        RPYB_CUDA(cudaGetLastError());
        return RPYB_OK;
    };
    return dtype == RPYB_F64 ? go(double{}) : go(float{});
}

RPYB_API int rpyb_ft_adjoint_left_mul(int dtype, int32_t width, int32_t depth, int64_t batch,
                                      void* out, const void* op, const void* arg, int64_t ld_out,
                                      int64_t ld_op, int64_t ld_arg, const int32_t* deg,
                                      void* stream)
{
    return adjoint_left_mul(dtype, width, depth, batch, out, op, arg, ld_out, ld_op, ld_arg, deg,
                            true, stream);
}

RPYB_API int rpyb_ft_adjoint_left_mul_fresh(int dtype, int32_t width, int32_t depth,
                                            int64_t batch, void* out, const void* op,
                                            const void* arg, int64_t ld_out, int64_t ld_op,
                                            int64_t ld_arg, const int32_t* deg, void* stream)
{
    return adjoint_left_mul(dtype, width, depth, batch, out, op, arg, ld_out, ld_op, ld_arg, deg,
                            false, stream);
}

RPYB_API int rpyb_sparse_map(int dtype, int64_t n_rows, int64_t n_cols, int64_t batch,
                             const int64_t* indptr, const int64_t* indices, const double* values,
                             void* y, const void* x, int64_t ld_y, int64_t ld_x, double scale,
                             void* stream)
{
    if (dtype != RPYB_F32 && dtype != RPYB_F64) return fail(RPYB_E_INVALID, "unsupported dtype");
    if (n_rows < 0 || n_cols < 0 || batch < 0) return fail(RPYB_E_INVALID, "negative size");
    if (batch == 0 || n_rows == 0) return RPYB_OK;
    if (!indptr || !y || !x) return fail(RPYB_E_INVALID, "null pointer");
    if (batch > 1 && (ld_y < n_rows || ld_x < n_cols))
        return fail(RPYB_E_INVALID, "row stride smaller than the vector size");
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    const int threads = 256;
    const unsigned blocks = grid_for(n_rows * batch, threads);
    if (dtype == RPYB_F64)
        csr_map_kernel<double><<<blocks, threads, 0, s>>>(n_rows, n_cols, batch, indptr, indices, values,
                                                         static_cast<double*>(y),
                                                         static_cast<const double*>(x), ld_y,
                                                         ld_x, scale);
    else
        csr_map_kernel<float><<<blocks, threads, 0, s>>>(n_rows, n_cols, batch, indptr, indices, values,
                                                        static_cast<float*>(y),
                                                        static_cast<const float*>(x), ld_y, ld_x,
                                                        scale);
    RPYB_CUDA(cudaGetLastError());
    return RPYB_OK;
}

}  // extern "C"
