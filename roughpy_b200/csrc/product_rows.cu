// Row-resident product: out (+)= lhs (x) rhs with a row's lower levels in
// shared memory (sm_100a).
//
// The top level holds most of a row's words, and each of its words needs the
// two top-level words L_N, R_N (and the old out_N), read once, and products of
// lower-level words.  One block stages the lower levels of both factors as
// float64 (a float32 word is converted once, not once a use), computes the
// lower output levels from them and streams the top level: coalesced reads and
// writes, all other operands from shared memory (split_unit).  The terms of a
// word are added in the same order as in the product kernels that read their
// operands through L1, so results are the same bits.
//
// Measured on B200 against the kernels that read lower levels through L1 (in
// product.cu, kept for shapes that do not fit and for bounded products): out =
// lhs (x) rhs, (5,6) float64 x 700 107 -> 61 us (5.4 TB/s), (7,5) float32 x 700
// 80 -> 41 us, (8,5) float32 107 -> 74 us, (8,3) float64 x 20000 145 -> 45 us
// (6.3 TB/s); accumulating, (2,12) float32 x 1024 57.5 -> 49.5 us, (4,7)
// float64 x 1000 130 -> 118 us.  What bounds it is HBM for float64 and short
// rows; for narrow float32 rows the shared-memory requests of the splits.
//
// out may be lhs (in place): the lower levels are staged before a word is
// written, and a top-level word of a factor is read only by the thread that
// then writes the same word.
#include <algorithm>

#include "product.cuh"
#include "row_units.cuh"

namespace rpyb {
namespace {

// dynamic shared memory a block may take (227 KB less the static part)
constexpr int64_t kRowSmem = 226 * 1024;
constexpr int64_t kRowSmemMost = kRowSmem + 64;   // with stage_room's padding
constexpr int kRowThreads = 1024;   // most threads a block

struct RowArgs {
    int width, top;
    int64_t db[kMaxDepth + 2];
    int64_t pw[kMaxDepth + 1];
    void* out;
    const void* lhs;
    const void* rhs;
    int64_t ld_out, ld_lhs, ld_rhs, batch;
    const int64_t* out_idx;
    const int64_t* lhs_idx;
    const int64_t* rhs_idx;
};

// The deepest top level of width D whose lower levels fit, both factors'.
template <int D>
constexpr int row_max_top()
{
    int64_t words = 0, pw = 1;
    for (int k = 0; k <= kMaxDepth; ++k) {   // words: below level k
        if (2 * words * 8 > kRowSmem) return k - 1;
        words += pw;
        pw *= D;
    }
    return kMaxDepth;
}

// Starts the lines of `runs` (at most 16) runs of `left` words (32 at most are
// wanted), `run` words apart from p, towards L2: one line a lane.
template <typename T>
__device__ __forceinline__ void prefetch_runs(const T* p, int64_t run, int runs, int64_t left,
                                              int lane)
{
    constexpr int kLines = sizeof(T) == 8 ? 2 : 1;   // of 128 bytes, a run
    if (lane < runs * kLines && (lane % kLines) * 16 < left)
        asm volatile("prefetch.global.L2 [%0];" ::"l"(p + (lane / kLines) * run + (lane % kLines) * 16));
}

template <typename T, typename TR, bool ACCUM, int D, int F>
__global__ void __launch_bounds__(kRowThreads, 1)
product_rows_kernel(const RowArgs a)
{
    constexpr int DD = D > 0 ? D : 1;
    constexpr int U = D > 0 ? Power<DD, F>::value : 16;
    extern __shared__ __align__(16) unsigned char row_smem[];
    const int N = a.top;
    const int d = D > 0 ? D : a.width;
    const int uu = D > 0 ? U : d;   // words a unit has
    const int TL = (int)a.db[N];
    double* const l_room = reinterpret_cast<double*>(row_smem);
    double* const r_room = l_room + stage_room(TL);
    const int tid = (int)threadIdx.x, B = (int)blockDim.x;
    const int lane = tid & 31, warp = tid >> 5, nwarps = B >> 5;

    for (int64_t b = blockIdx.y; b < a.batch; b += gridDim.y) {
        // not restrict: out may be lhs
        T* out = static_cast<T*>(a.out) + (a.out_idx ? a.out_idx[b] : b) * a.ld_out;
        const T* lhs = static_cast<const T*>(a.lhs) + (a.lhs_idx ? a.lhs_idx[b] : b) * a.ld_lhs;
        const TR* rhs = static_cast<const TR*>(a.rhs) + (a.rhs_idx ? a.rhs_idx[b] : b) * a.ld_rhs;
        __syncthreads();   // the previous row is done with the buffers
        const double* L = stage_words(l_room, lhs, TL, tid, B);
        const double* R = stage_words(r_room, rhs, TL, tid, B);
        // The top-level words of a warp's next task start towards L2 while it
        // works on one.  (The whole top level at once would be more than L2
        // holds over all resident rows: (6,5) float64 ran at 3.1 TB/s so.)
        const int top_tasks = N >= F ? (int)((a.pw[N - F] + 31) >> 5) : 0;
        const int tstep = nwarps * (int)gridDim.x;
        auto prefetch_task = [&](int t) {
            if (t >= top_tasks) return;
            const int64_t run = a.pw[N - F];
            const int64_t o = a.db[N] + t * 32;
            const int64_t left = run - t * 32;
            prefetch_runs(lhs + o, run, uu, left, lane);
            prefetch_runs(rhs + o, run, uu, left, lane);
            if (ACCUM) prefetch_runs(static_cast<const T*>(out) + o, run, uu, left, lane);
        };
        prefetch_task(warp + nwarps * (int)blockIdx.x);
        T out0 = T(0);
        if (ACCUM && tid == 0 && blockIdx.x == 0) out0 = out[0];
        asm volatile("cp.async.wait_all;" ::: "memory");
        __syncthreads();
        const double l0 = L[0], r0 = R[0];

        // unit r of the top level (streamed) or of a lower one (in shared memory)
        auto unit = [&](auto kc, auto topc, uint32_t r) {
            constexpr int K = decltype(kc)::value;
            constexpr bool TOP = decltype(topc)::value;
            constexpr int run = Power<DD, K - F>::value, begin = LevelStart<DD, K>::value;
            if (run % 32 != 0 && r >= (uint32_t)run) return;
            double acc[U];
            T* op = out + begin + r;
#pragma unroll
            for (int u = 0; u < U; ++u) acc[u] = ACCUM ? (double)op[u * run] : 0.0;
            if constexpr (TOP) {
                const T* lp = lhs + begin + r;
                T lv[U];
#pragma unroll
                for (int u = 0; u < U; ++u) lv[u] = lp[u * run];
#pragma unroll
                for (int u = 0; u < U; ++u) acc[u] = fma((double)lv[u], r0, acc[u]);
            } else {
                const double* lp = L + begin + r;
#pragma unroll
                for (int u = 0; u < U; ++u) acc[u] = fma(lp[u * run], r0, acc[u]);
            }
            if constexpr (TOP) {
                const TR* rp = rhs + begin + r;
                TR rv[U];   // in flight during the splits
#pragma unroll
                for (int u = 0; u < U; ++u) rv[u] = rp[u * run];
                split_unit<DD, F, K, U>(acc, L, R, r);
#pragma unroll
                for (int u = 0; u < U; ++u) acc[u] = fma(l0, (double)rv[u], acc[u]);
            } else {
                split_unit<DD, F, K, U>(acc, L, R, r);
                const double* rp = R + begin + r;
#pragma unroll
                for (int u = 0; u < U; ++u) acc[u] = fma(l0, rp[u * run], acc[u]);
            }
#pragma unroll
            for (int u = 0; u < U; ++u) op[u * run] = (T)acc[u];
        };
        auto any_unit = [&](int k, uint32_t r) {
            const uint32_t run = (uint32_t)a.pw[k - 1];
            if (r >= run) return;
            const int o = (int)a.db[k] + (int)r;
            double acc[16];
#pragma unroll
            for (int u = 0; u < 16; ++u) {
                if (u >= d) break;
                acc[u] = ACCUM ? (double)out[o + u * run] : 0.0;
                acc[u] = fma(k < N ? L[o + u * run] : (double)lhs[o + u * run], r0, acc[u]);
            }
            split_unit_any(acc, L, R, a.db, a.pw, (uint32_t)d, k, r);
#pragma unroll
            for (int u = 0; u < 16; ++u) {
                if (u >= d) break;
                const double rv = k < N ? R[o + u * run] : (double)rhs[o + u * run];
                out[o + u * run] = (T)fma(l0, rv, acc[u]);
            }
        };
        // levels 0 and below the owned letters, word by word
        auto short_levels = [&]() {
            for (int k = 1; k < F && k <= N; ++k) {
                for (int w = lane; w < (int)a.pw[k]; w += 32) {
                    const int o = (int)a.db[k] + w;
                    double v = ACCUM ? (double)out[o] : 0.0;
                    v = fma(k < N ? L[o] : (double)lhs[o], r0, v);
                    int ds = 1;
                    for (int s = 1; s < k; ++s) {
                        ds *= d;
                        v = fma(L[a.db[k - s] + w / ds], R[a.db[s] + w % ds], v);
                    }
                    out[o] = (T)fma(l0, k < N ? R[o] : (double)rhs[o], v);
                }
            }
        };

        int t = warp;
        const int step = nwarps;
        if (N >= F) {
            for (t += nwarps * (int)blockIdx.x; t < top_tasks; t += tstep) {
                prefetch_task(t + tstep);
                const uint32_t r = (uint32_t)(t * 32 + lane);
                if constexpr (D > 0) {
                    with_level<F, row_max_top<DD>()>(N, [&](auto kc) {
                        unit(kc, std::integral_constant<bool, true>{}, r);
                    });
                } else {
                    any_unit(N, r);
                }
            }
            t = gridDim.x > 1 ? warp : t - top_tasks;
        }
        if (blockIdx.x != 0) continue;
        for (int k = max(N - 1, F - 1); k >= F - 1;) {   // level F - 1: the short levels' task
            const int tasks = k >= F ? (int)((a.pw[k - F] + 31) >> 5) : 1;
            if (t >= tasks) {
                t -= tasks;
                --k;
                continue;
            }
            if (k < F) {
                short_levels();
            } else {
                const uint32_t r = (uint32_t)(t * 32 + lane);
                if constexpr (D > 0) {
                    with_level<F, row_max_top<DD>() - 1>(k, [&](auto kc) {
                        unit(kc, std::integral_constant<bool, false>{}, r);
                    });
                } else {
                    any_unit(k, r);
                }
            }
            t += step;
        }
        if (tid == 0) out[0] = out0 + (T)l0 * (T)r0;   // level 0, in the rows' type
    }
}

// The top level of rows whose lower levels do not fit but whose next lower
// level's do (width 8 depth 6, 4 and 8, 5 and 7, ...), in slabs: a block takes
// the words (u, a, rho) of one second letter a, all first letters u and the
// N - 2 letters rho.  With 2 <= p < N their left words are L_p[u, a, ..], a
// d-th of each level, and their right words the levels R_1 .. R_{N-2}, so both
// are staged as float64 as before; L_p's part is as many words as level p - 1,
// and in that place split_unit sees a product of depth N - 1.  Left over are
// p = 1, whose right words R_{N-1}[a, rho] are one run, and the streamed ends.
// Levels below N are a row-resident product of their own.  Measured on B200, (8,6)
// float32 x 1024 accumulating, calls in a row: 1159 -> 1106 us, at the board's
// power cap (SM clock 1965 -> 1665 MHz); in bursts of 20, 1006 us (4.9 TB/s).  In
// place (8,6) float32 x 500 1.16 -> 0.47 ms.  What bounds it is the latency of the
// streamed words at 27 warps an SM (64 registers a thread): 53 % DRAM, 47 % of the
// shared-memory wavefronts, 37 % issue.
template <typename T, typename TR, bool ACCUM, int D>
__global__ void __launch_bounds__(kRowThreads, 1)
product_slab_kernel(const RowArgs a)
{
    constexpr int U = D;
    extern __shared__ __align__(16) unsigned char row_smem[];
    __shared__ double first[D];   // L_1
    const int N = a.top;
    const int TL = (int)a.db[N - 1];   // words below level N - 1
    double* const l_room = reinterpret_cast<double*>(row_smem);
    double* const r_room = l_room + stage_room(TL);
    const int tid = (int)threadIdx.x, B = (int)blockDim.x;
    const int lane = tid & 31, warp = tid >> 5, nwarps = B >> 5;
    const uint32_t letter = blockIdx.x;
    const uint32_t rho_n = (uint32_t)a.pw[N - 2], run = (uint32_t)a.pw[N - 1];

    for (int64_t b = blockIdx.y; b < a.batch; b += gridDim.y) {
        T* out = static_cast<T*>(a.out) + (a.out_idx ? a.out_idx[b] : b) * a.ld_out;
        const T* lhs = static_cast<const T*>(a.lhs) + (a.lhs_idx ? a.lhs_idx[b] : b) * a.ld_lhs;
        const TR* rhs = static_cast<const TR*>(a.rhs) + (a.rhs_idx ? a.rhs_idx[b] : b) * a.ld_rhs;
        __syncthreads();   // the previous row is done with the buffers
        const double* R = stage_words(r_room, rhs, TL, tid, B);
        for (int j = 1; j <= N - 2; ++j) {
            // level j's place: L_{j+1}[u, letter, ..]
            const uint32_t n = (uint32_t)a.pw[j], part = (uint32_t)a.pw[j - 1];
            const T* src = lhs + a.db[j + 1] + (int64_t)letter * part;
            double* dst = l_room + a.db[j];
            constexpr int kLoads = 8;
            for (uint32_t i0 = tid; i0 < n; i0 += kLoads * B) {
                T v[kLoads];
#pragma unroll
                for (int k = 0; k < kLoads; ++k) {
                    const uint32_t i = i0 + k * B, u = i / part;
                    v[k] = i < n ? src[(int64_t)u * n + (i - u * part)] : T(0);
                }
#pragma unroll
                for (int k = 0; k < kLoads; ++k)
                    if (i0 + k * B < n) dst[i0 + k * B] = (double)v[k];
            }
        }
        if (tid < D) first[tid] = (double)lhs[1 + tid];
        const int tasks = (int)((rho_n + 31) >> 5);
        const int64_t begin = a.db[N] + (int64_t)letter * rho_n;
        auto prefetch_task = [&](int t) {
            if (t >= tasks) return;
            const int64_t left = rho_n - t * 32;
            prefetch_runs(lhs + begin + t * 32, run, D, left, lane);
            prefetch_runs(rhs + begin + t * 32, run, D, left, lane);
            prefetch_runs(rhs + a.db[N - 1] + (int64_t)letter * rho_n + t * 32, run, 1, left, lane);
            if (ACCUM) prefetch_runs(static_cast<const T*>(out) + begin + t * 32, run, D, left, lane);
        };
        prefetch_task(warp);
        asm volatile("cp.async.wait_all;" ::: "memory");
        __syncthreads();
        const double l0 = (double)lhs[0], r0 = R[0];
        with_level<1, row_max_top<D>()>(N - 1, [&](auto kc) {
            constexpr int K = decltype(kc)::value;   // depth of what split_unit sees
            constexpr int RHO = Power<D, K - 1>::value, RUN = Power<D, K>::value;
            for (int t = warp; t < tasks; t += nwarps) {
                prefetch_task(t + nwarps);
                const uint32_t rho = (uint32_t)(t * 32 + lane);
                if (RHO % 32 != 0 && rho >= (uint32_t)RHO) continue;
                T* op = out + begin + rho;
                const T* lp = lhs + begin + rho;
                const TR* rp = rhs + begin + rho;
                T av[U], lv[U];
#pragma unroll
                for (int u = 0; u < U; ++u) {
                    if (ACCUM) av[u] = op[(int64_t)u * RUN];
                    lv[u] = lp[(int64_t)u * RUN];
                }
                double acc[U];
#pragma unroll
                for (int u = 0; u < U; ++u) acc[u] = fma((double)lv[u], r0, ACCUM ? (double)av[u] : 0.0);
                TR rv[U];   // in flight during the splits
#pragma unroll
                for (int u = 0; u < U; ++u) rv[u] = rp[(int64_t)u * RUN];
                const double x1 = (double)rhs[LevelStart<D, K>::value + (int64_t)letter * RHO + rho];
                split_unit<D, 1, K, U>(acc, l_room, R, rho);
#pragma unroll
                for (int u = 0; u < U; ++u) acc[u] = fma(first[u], x1, acc[u]);
#pragma unroll
                for (int u = 0; u < U; ++u) op[(int64_t)u * RUN] = (T)fma(l0, (double)rv[u], acc[u]);
            }
        });
    }
}

using RowFn = void (*)(RowArgs);

template <typename T, typename TR, bool ACCUM>
RowFn row_fn(int width)
{
    switch (width) {
        case 2: return &product_rows_kernel<T, TR, ACCUM, 2, 3>;
        case 3: return &product_rows_kernel<T, TR, ACCUM, 3, 2>;
        case 4: return &product_rows_kernel<T, TR, ACCUM, 4, 1>;
        case 5: return &product_rows_kernel<T, TR, ACCUM, 5, 1>;
        case 6: return &product_rows_kernel<T, TR, ACCUM, 6, 1>;
        case 7: return &product_rows_kernel<T, TR, ACCUM, 7, 1>;
        case 8: return &product_rows_kernel<T, TR, ACCUM, 8, 1>;
        default: return &product_rows_kernel<T, TR, ACCUM, 0, 1>;
    }
}

template <typename T, typename TR, bool ACCUM>
RowFn slab_fn(int width)
{
    switch (width) {
        case 4: return &product_slab_kernel<T, TR, ACCUM, 4>;
        case 5: return &product_slab_kernel<T, TR, ACCUM, 5>;
        case 6: return &product_slab_kernel<T, TR, ACCUM, 6>;
        case 7: return &product_slab_kernel<T, TR, ACCUM, 7>;
        case 8: return &product_slab_kernel<T, TR, ACCUM, 8>;
        default: return nullptr;
    }
}

RowArgs row_args(const Geometry& g, int top, const ProductRows& rows)
{
    RowArgs a{};
    a.width = g.width;
    a.top = top;
    for (int k = 0; k <= kMaxDepth + 1; ++k) a.db[k] = g.db[k];
    for (int k = 0; k <= kMaxDepth; ++k) a.pw[k] = g.pw[k];
    a.out = rows.out;
    a.lhs = rows.lhs;
    a.rhs = rows.rhs;
    a.ld_out = rows.ld_out;
    a.ld_lhs = rows.ld_lhs;
    a.ld_rhs = rows.ld_rhs;
    a.batch = rows.batch;
    a.out_idx = rows.out_idx;
    a.lhs_idx = rows.lhs_idx;
    a.rhs_idx = rows.rhs_idx;
    return a;
}

// whether the spec is the whole truncated product of whole rows
bool whole_product(const ProductSpec& spec, const ProductRows& rows)
{
    if (spec.klo != 1 || !spec.lhs0_from_mem || spec.lhs0_add != 0.0 || rows.addend) return false;
    if (!spec.l0_write || !spec.l0_prod || spec.l0_const != 0.0 || spec.scale0 != 1.0 ||
        spec.l0_base != (spec.accumulate ? 1 : 0))
        return false;
    for (int k = 1; k <= spec.khi; ++k)
        if (spec.pmin[k] != 0 || spec.pmax[k] != k || spec.scale[k] != 1.0) return false;
    return true;
}

}  // namespace

bool product_rows_available(const Geometry& g, const ProductSpec& spec, const ProductRows& rows)
{
    const int N = spec.khi;
    if (g.width < 2 || g.width > 16 || N < 1 || 2 * g.db[N] * 8 > kRowSmem) return false;
    return whole_product(spec, rows);
}

int launch_product_rows(int dtype, const Geometry& g, const ProductSpec& spec,
                        const ProductRows& rows, bool in_place, cudaStream_t stream)
{
    RowArgs a = row_args(g, spec.khi, rows);
    RowFn fn;
    if (dtype == RPYB_F64)
        fn = spec.accumulate ? row_fn<double, double, true>(g.width) : row_fn<double, double, false>(g.width);
    else if (dtype == kMixedF64F32)
        fn = spec.accumulate ? row_fn<double, float, true>(g.width) : row_fn<double, float, false>(g.width);
    else
        fn = spec.accumulate ? row_fn<float, float, true>(g.width) : row_fn<float, float, false>(g.width);
    const int F = g.width == 2 ? 3 : g.width == 3 ? 2 : 1;
    const size_t smem = (size_t)(2 * stage_room((int)g.db[a.top]) * 8);
    const int64_t units = a.top >= F ? g.pw[a.top - F] : g.pw[a.top];
    int64_t threads = row_block_threads(g, a.top, F, smem, kRowSmem, rows.batch, kRowThreads);
    // fewer rows than SMs: blocks share a row's top level (not in place, where
    // one block would write lower levels that another still has to stage)
    int64_t slices = 1;
    if (!in_place && rows.batch < 148) {
        // (every block stages the lower levels: with enough threads to have
        // them all in flight at once)
        const int64_t least = std::max<int64_t>(128, g.db[a.top] / 8);
        slices = std::max<int64_t>(1, std::min<int64_t>({16, 148 / rows.batch, units / least}));
        if (slices > 1)
            threads = std::min<int64_t>(threads, (units + 32 * slices - 1) / (32 * slices) * 32);
    }
    const dim3 grid((unsigned)slices, (unsigned)std::min<int64_t>(rows.batch, 65535), 1);
    if (int rc = allow_shared_memory(fn, smem, kRowSmemMost)) return rc;
    fn<<<grid, (unsigned)threads, smem, stream>>>(a);
    RPYB_CUDA(cudaGetLastError());
    return RPYB_OK;
}

bool product_slabs_available(const Geometry& g, const ProductSpec& spec, const ProductRows& rows)
{
    const int N = spec.khi;
    return g.width >= 4 && g.width <= 8 && N >= 3 && 2 * g.db[N] * 8 > kRowSmem &&
           2 * g.db[N - 1] * 8 <= kRowSmem && whole_product(spec, rows);
}

int launch_product_slabs(int dtype, const Geometry& g, const ProductSpec& spec,
                         const ProductRows& rows, bool in_place, cudaStream_t stream)
{
    const RowArgs a = row_args(g, spec.khi, rows);
    RowFn fn;
    if (dtype == RPYB_F64)
        fn = spec.accumulate ? slab_fn<double, double, true>(g.width) : slab_fn<double, double, false>(g.width);
    else if (dtype == kMixedF64F32)
        fn = spec.accumulate ? slab_fn<double, float, true>(g.width) : slab_fn<double, float, false>(g.width);
    else
        fn = spec.accumulate ? slab_fn<float, float, true>(g.width) : slab_fn<float, float, false>(g.width);
    const size_t smem = (size_t)(2 * stage_room((int)g.db[a.top - 1]) * 8);
    const int64_t threads = row_block_threads(g, a.top - 1, 1, smem, kRowSmem, rows.batch * g.width, kRowThreads);
    if (int rc = allow_shared_memory(fn, smem, kRowSmemMost)) return rc;
    const dim3 grid((unsigned)g.width, (unsigned)std::min<int64_t>(rows.batch, 65535), 1);
    // the top level first: in place, the lower levels it reads are still the old ones
    fn<<<grid, (unsigned)threads, smem, stream>>>(a);
    RPYB_CUDA(cudaGetLastError());
    ProductSpec low = spec;
    low.khi = spec.khi - 1;
    return launch_product_rows(dtype, g, low, rows, in_place, stream);
}

}  // namespace rpyb
