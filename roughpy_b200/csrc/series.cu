// exp, fmexp and log of dense free tensors with the whole Horner series of a
// row in one block (sm_100a).
//
// The series R <- base + scale_s (c_s + R) (x) x (free_tensor_exp.hpp:26-35,
// free_tensor_fmexp.hpp:31-38, free_tensor_log.hpp:23-38) runs N steps, and
// step s reaches level s only.  So the top level, most of the words, is
// computed once, in the last step, from the levels below it:
//
//   out_N[w] = base_N[w] + scale (c x_N[w] + sum_{0<p<N} R_p (x) x_{N-p}),
//
// with x_N read and out_N written once, coalesced, and everything else in
// shared memory as float64: the lower levels of x, and R's in two buffers.
// What a row cannot do without is one read of x and one write of out.
// As one product launch per step (the only form before, kept for shapes whose
// lower levels do not fit), a row moved N + 1 times through memory, with
// float32 rows widened to float64 copies for log.  Measured on B200, whole call
// with the zero fill of its result, before -> after: exp (5,5) float32, 4001
// rows 242 -> 59 us; log (6,5), 4096 rows, float64 322 -> 174 us, float32
// 645 -> 107 us; exp (2,12) float32, 1024 rows 201 -> 93 us; exp (6,6) float64,
// 600 rows 246 -> 183 us; log (2,6) float64, 200000 rows 2.73 -> 0.58 ms.
//
// A thread owns U = D^F words u * d^(k-F) + r of a level, u over the first F
// letters, for one suffix r; lanes take consecutive r, so right-factor words
// x[r mod d^s] are conflict-free runs and left-factor words R[u, r / d^s]
// broadcasts or short runs: U + 1 shared loads feed U FMAs, which at U >= 4
// keeps the shared-memory pipe, this kernel's second bound after HBM, within
// 1.25 requests an FMA.  Levels are compile-time constants inside a unit.
#include "series.cuh"

#include "row_units.cuh"

#include <algorithm>

namespace rpyb {
namespace {

// dynamic shared memory a block may take (227 KB less the static part)
constexpr int64_t kSeriesSmem = 226 * 1024;
constexpr int kSeriesThreads = 1024;   // most threads a block

struct SeriesArgs {
    int width, top, arg_max;
    bool fresh;                    // log: out[0] counts as zero
    double coeff[kMaxDepth + 1];   // 1 / deg, or log's series coefficient
    int64_t db[kMaxDepth + 2];
    int64_t pw[kMaxDepth + 1];
    void* out;
    const void* arg;
    const void* mult;
    int64_t ld_out, ld_arg, ld_mult, batch;
};

// The deepest top level of width D whose lower levels fit (three copies).
template <int D>
constexpr int series_max_top()
{
    int64_t words = 0, pw = 1;
    for (int k = 0; k <= kMaxDepth; ++k) {   // words: below level k
        if (3 * words * 8 > kSeriesSmem) return k - 1;
        words += pw;
        pw *= D;
    }
    return kMaxDepth;
}

// One step's work is dealt to warps in tasks of 32 units of one level, the
// highest level first (the levels shorter than the owned letters are the last
// task), so that a step's critical path is a few units whatever the depth.
template <typename T, SeriesKind KIND, int D, int F>
__global__ void __launch_bounds__(kSeriesThreads, 1)
series_kernel(const SeriesArgs a)
{
    constexpr int DD = D > 0 ? D : 1;
    constexpr int U = D > 0 ? Power<DD, F>::value : 16;
    constexpr bool MULT = KIND == kSeriesFmexp;
    constexpr bool SCALE = KIND != kSeriesLog;
    extern __shared__ __align__(16) unsigned char series_smem[];
    const int N = a.top;
    const int d = D > 0 ? D : a.width;
    const int TL = (int)a.db[N];
    double* X = reinterpret_cast<double*>(series_smem);
    double* Rc = X + TL;
    double* Rn = Rc + TL;
    const int tid = (int)threadIdx.x, B = (int)blockDim.x;
    const int lane = tid & 31, warp = tid >> 5, nwarps = B >> 5;

    for (int64_t b = blockIdx.y; b < a.batch; b += gridDim.y) {
        T* __restrict__ out = static_cast<T*>(a.out) + b * a.ld_out;
        const T* __restrict__ arg = static_cast<const T*>(a.arg) + b * a.ld_arg;
        const T* __restrict__ mult =
            MULT ? static_cast<const T*>(a.mult) + b * a.ld_mult : nullptr;
        const int xend = (int)min(a.db[N], a.db[a.arg_max + 1]);   // x's words below the top
        const bool xtop = a.arg_max >= N;
        __syncthreads();   // the previous row is done with the buffers
        constexpr int kLoads = 8;   // independent loads in flight a thread
        for (int i0 = tid; i0 < TL; i0 += kLoads * B) {
            T v[kLoads];
#pragma unroll
            for (int j = 0; j < kLoads; ++j)
                v[j] = i0 + j * B < xend ? __ldg(arg + i0 + j * B) : T(0);
#pragma unroll
            for (int j = 0; j < kLoads; ++j)
                if (i0 + j * B < TL) X[i0 + j * B] = (double)v[j];
        }
        if (xtop && blockIdx.x == 0) {
            // the top level, read in the last step, starts towards L2 now
            const char* p = reinterpret_cast<const char*>(arg + a.db[N]);
            const int64_t bytes = a.pw[N] * (int64_t)sizeof(T);
            for (int64_t l = (int64_t)tid * 128; l < bytes; l += (int64_t)B * 128)
                asm volatile("prefetch.global.L2 [%0];" ::"l"(p + l));
        }
        const double c_fm = MULT ? (double)__ldg(mult) : 1.0;
        const double c_in = KIND == kSeriesLog && !a.fresh ? (double)out[0] : 0.0;
        __syncthreads();

        for (int s = 1; s <= N; ++s) {
            const bool last = s == N;
            // this step's scalar of R and the factor of its product
            double c = c_fm;
            if constexpr (KIND == kSeriesLog) {
                c = a.coeff[N - s + 1];
                if (s == 1) c += c_in;
            }
            const double scale = SCALE ? a.coeff[N - s + 1] : 1.0;
            // lane's unit r of level k < N: R's next words, or the result's
            auto low_unit = [&](auto kc, uint32_t r) {
                constexpr int K = decltype(kc)::value;
                constexpr int run = Power<DD, K - F>::value, begin = LevelStart<DD, K>::value;
                if (run % 32 != 0 && r >= (uint32_t)run) return;
                double acc[U];
                const double* xp = X + begin + r;
#pragma unroll
                for (int u = 0; u < U; ++u) acc[u] = c * xp[u * run];
                split_unit<DD, F, K, U>(acc, Rc, X, r);
                if constexpr (SCALE) {
#pragma unroll
                    for (int u = 0; u < U; ++u) acc[u] *= scale;
                }
                if constexpr (MULT) {
                    const T* mp = mult + begin + r;
#pragma unroll
                    for (int u = 0; u < U; ++u) acc[u] += (double)__ldg(mp + u * run);
                }
                if (last) {
                    T* op = out + begin + r;
#pragma unroll
                    for (int u = 0; u < U; ++u) op[u * run] = (T)acc[u];
                } else {
                    double* rp = Rn + begin + r;
#pragma unroll
                    for (int u = 0; u < U; ++u) rp[u * run] = acc[u];
                }
            };
            // lane's unit r of the top level: x_N in, out_N out
            auto top_unit = [&](auto kc, uint32_t r) {
                constexpr int K = decltype(kc)::value;
                constexpr int run = Power<DD, K - F>::value, begin = LevelStart<DD, K>::value;
                if (run % 32 != 0 && r >= (uint32_t)run) return;
                T xv[U];   // in flight during the splits
                const T* ap = arg + begin + r;
#pragma unroll
                for (int u = 0; u < U; ++u) xv[u] = xtop ? __ldg(ap + u * run) : T(0);
                double acc[U];
#pragma unroll
                for (int u = 0; u < U; ++u) acc[u] = 0.0;
                split_unit<DD, F, K, U>(acc, Rc, X, r);
                T* op = out + begin + r;
#pragma unroll
                for (int u = 0; u < U; ++u) {
                    double v = fma(c, (double)xv[u], acc[u]);
                    if constexpr (SCALE) v *= scale;
                    if constexpr (MULT) v += (double)__ldg(mult + begin + r + u * run);
                    op[u * run] = (T)v;
                }
            };
            // the same for a runtime width, both kinds of level
            auto any_unit = [&](int k, uint32_t r) {
                const uint32_t run = (uint32_t)a.pw[k - 1];
                if (r >= run) return;
                const int o = (int)a.db[k] + (int)r;
                double acc[16];
#pragma unroll
                for (int u = 0; u < 16; ++u)
                    if (u < d)
                        acc[u] = c * (k < N ? X[o + u * run] : xtop ? (double)__ldg(arg + o + u * run) : 0.0);
                split_unit_any(acc, Rc, X, a.db, a.pw, (uint32_t)d, k, r);
#pragma unroll
                for (int u = 0; u < 16; ++u) {
                    if (u >= d) break;
                    double v = acc[u];
                    if constexpr (SCALE) v *= scale;
                    if constexpr (MULT) v += (double)__ldg(mult + o + u * run);
                    if (last) out[o + u * run] = (T)v;
                    else Rn[o + u * run] = v;
                }
            };
            // the words of the levels below the owned letters, one by one
            auto short_levels = [&]() {
                for (int k = 1; k < F && k <= s; ++k) {
                    for (int w = lane; w < (int)a.pw[k]; w += 32) {
                        const int o = (int)a.db[k] + w;
                        double v = c * (k < N ? X[o] : xtop ? (double)__ldg(arg + o) : 0.0);
                        int ds = 1;
                        for (int t = 1; t < k; ++t) {
                            ds *= d;
                            v = fma(Rc[a.db[k - t] + w / ds], X[a.db[t] + w % ds], v);
                        }
                        if constexpr (SCALE) v *= scale;
                        if constexpr (MULT) v += (double)__ldg(mult + o);
                        if (last) out[o] = (T)v;
                        else Rn[o] = v;
                    }
                }
            };
            int t = warp, step = nwarps, k = min(s, N - 1);
            if (last && N >= F) {
                // the top level is shared by the row's blocks
                const int top_tasks = (int)((a.pw[N - F] + 31) >> 5);
                step = nwarps * (int)gridDim.x;
                for (t += nwarps * (int)blockIdx.x; t < top_tasks; t += step) {
                    const uint32_t r = (uint32_t)(t * 32 + lane);
                    if constexpr (D > 0) {
                        with_level<F, series_max_top<DD>()>(N, [&](auto kc) { top_unit(kc, r); });
                    } else {
                        any_unit(N, r);
                    }
                }
                // the lower levels are the first block's: they carry on the
                // count of tasks, or start anew where blocks share the row
                t = gridDim.x > 1 ? warp : t - top_tasks;
                step = nwarps;
            }
            if (!last || blockIdx.x == 0) {
                for (k = max(k, F - 1); k >= F - 1;) {   // level F - 1: the short levels' task
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
                            with_level<F, series_max_top<DD>() - 1>(k, [&](auto kc) { low_unit(kc, r); });
                        } else {
                            any_unit(k, r);
                        }
                    }
                    t += step;
                }
            }
            if (last) {
                if (tid == 0 && blockIdx.x == 0) out[0] = KIND == kSeriesLog ? T(0) : (T)c_fm;
            } else {
                __syncthreads();
                double* tmp = Rc;
                Rc = Rn;
                Rn = tmp;
            }
        }
    }
}

using SeriesFn = void (*)(SeriesArgs);

// first letters a unit owns: enough for four words or more a unit
int series_first(int width) { return width == 2 ? 3 : width == 3 ? 2 : 1; }

template <typename T, SeriesKind KIND>
SeriesFn series_fn(int width)
{
    switch (width) {
        case 2: return &series_kernel<T, KIND, 2, 3>;
        case 3: return &series_kernel<T, KIND, 3, 2>;
        case 4: return &series_kernel<T, KIND, 4, 1>;
        case 5: return &series_kernel<T, KIND, 5, 1>;
        case 6: return &series_kernel<T, KIND, 6, 1>;
        case 7: return &series_kernel<T, KIND, 7, 1>;
        case 8: return &series_kernel<T, KIND, 8, 1>;
        default: return &series_kernel<T, KIND, 0, 1>;
    }
}

template <typename T>
SeriesFn series_fn(SeriesKind kind, int width)
{
    switch (kind) {
        case kSeriesExp: return series_fn<T, kSeriesExp>(width);
        case kSeriesFmexp: return series_fn<T, kSeriesFmexp>(width);
        default: return series_fn<T, kSeriesLog>(width);
    }
}

}  // namespace

bool series_available(const Geometry& g, int top)
{
    return g.width >= 2 && g.width <= 16 && top >= 1 && 3 * g.db[top] * 8 <= kSeriesSmem;
}

// The longest rows that the runtime width takes, (13..16, 4), where a few of
// them leave most SMs idle: (16,4) float64, row-resident / launches on B200, log
// x 8 72 / 35 us, x 64 76 / 70, fmexp x 8 63 / 46, x 64 87 / 134; log of float32 x
// 32 66 / 78.  Float32 exp and fmexp stay: a launch a step rounds every step to
// float32.
bool series_slower(int dtype, SeriesKind kind, const Geometry& g, int top, int64_t batch)
{
    if (dtype == RPYB_F32 && kind != kSeriesLog) return false;
    return g.width > 12 && g.db[top] > 2000 && batch < (dtype == RPYB_F64 && kind == kSeriesLog ? 64 : 32);
}

int launch_series(int dtype, SeriesKind kind, const Geometry& g, int top, int arg_max,
                  const SeriesRows& rows, cudaStream_t stream)
{
    if (rows.batch <= 0) return RPYB_OK;
    SeriesArgs a{};
    a.width = g.width;
    a.top = top;
    a.arg_max = std::min(arg_max, top);
    a.fresh = rows.fresh;
    for (int deg = 1; deg <= top; ++deg)
        a.coeff[deg] = (kind == kSeriesLog && deg % 2 == 0) ? -(1.0 / deg) : 1.0 / deg;
    for (int k = 0; k <= kMaxDepth + 1; ++k) a.db[k] = g.db[k];
    for (int k = 0; k <= kMaxDepth; ++k) a.pw[k] = g.pw[k];
    a.out = rows.out;
    a.arg = rows.arg;
    a.mult = kind == kSeriesFmexp ? rows.mult : nullptr;
    a.ld_out = rows.ld_out;
    a.ld_arg = rows.ld_arg;
    a.ld_mult = rows.ld_mult;
    a.batch = rows.batch;

    const int first = series_first(g.width);
    SeriesFn fn = dtype == RPYB_F64 ? series_fn<double>(kind, g.width)
                                    : series_fn<float>(kind, g.width);
    const size_t smem = (size_t)(3 * g.db[top] * 8);
    const int64_t units = top >= first ? g.pw[top - first] : g.pw[top];
    const int64_t threads = row_block_threads(g, top, first, smem, kSeriesSmem, rows.batch, kSeriesThreads);
    // fewer rows than SMs: blocks of one row share its top level (each
    // computes the lower levels for itself).  Not for a log whose incoming
    // out[0] every block would have to read before one of them writes it.
    int64_t slices = 1;
    if ((kind != kSeriesLog || rows.fresh) && rows.batch < 148)
        slices = std::max<int64_t>(1, std::min<int64_t>({16, 296 / rows.batch, units / (2 * threads)}));
    const dim3 grid((unsigned)slices, (unsigned)std::min<int64_t>(rows.batch, 65535), 1);
    if (int rc = allow_shared_memory(fn, smem, kSeriesSmem)) return rc;
    fn<<<grid, (unsigned)threads, smem, stream>>>(a);
    RPYB_CUDA(cudaGetLastError());
    return RPYB_OK;
}

}  // namespace rpyb
