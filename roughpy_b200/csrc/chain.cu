// Fused chain products: acc[q] <- src[r_0] * src[r_1] * ... (the unit for an
// empty list), its float64 log, or the log's Hall coordinates, one block per
// row q, so that the running product never leaves the SM (sm_100a).
//
// Shared memory holds the running product whole, as float64, a second buffer
// for its lower levels, and the lower levels of the factor in use and of the
// next one, which is copied in while this one is multiplied.  Lower levels
// ping-pong between two buffers; the top level is updated in place, since a
// top-level word reads of its own operand only itself and lower levels.  The
// factor's top-level words are read where they are (queries share popular
// rows, which stay in L2) and start towards L2 when the query does.  Work is
// dealt to warps in tasks of 32 units of one level (split_unit), the top level
// first.  log(X) follows in the same buffers by the Horner steps of the
// float64 log (free_tensor_log.hpp:23-38), step s reaching level s, and the
// projection gathers through the packed tensor -> Lie map from the whole log
// in shared memory.
//
// The layout before kept the top level in registers (18 words a thread, one
// block of 512 an SM) and read every operand of a split through L1 in strided
// words: 1.39 ms for 8192 queries of at most four (6,5) factors, log and
// projection, on a 2^14-event float64 tree, against 1.06 ms here, where
// shared-memory wavefronts (73 % busy) and issue (54 %) bound it, the
// projection's gathers among them.  100000 such queries: 18.5 -> 14.0 ms with
// the host's dissection, 12.9 with the device's; 20000 at (5,5), which did not fit
// the registers, 4.9 -> 2.0 ms.  Up to a few hundred queries are a chain or two
// an SM, and there the registers were faster: 16 queries of 1024 events at (6,5),
// with their host time, 49 -> 55 us in float64 and 46 -> 61 in float32, whose
// factors have to be waited for and widened before a product.  (Holding the next
// factor's words in registers across a product took 3 us off a few float32
// queries and cost large batches 4 to 7 %.)
#include <algorithm>

#include "row_units.cuh"
#include "stream_ops.cuh"

namespace rpyb {
namespace {

constexpr int64_t kChainSmem = 226 * 1024;
constexpr int kChainThreads = 1024;   // most threads a block

struct ChainArgs {
    int64_t T = 0;
    int64_t db[kMaxDepth + 2] = {};
    int64_t pw[kMaxDepth + 1] = {};
    double coeff[kMaxDepth + 1] = {};       // (-1)^(deg+1) / deg
    int depth = 0;
    int64_t n = 0;
    const int64_t* off = nullptr;      // [n + 1] into rows, or (stride > 0) the
    const int64_t* rows = nullptr;     // source rows of q's off[q] factors at q * stride
    int64_t stride = 0;
    const void* src = nullptr;         // [*, T] factors (float or double)
    double* acc = nullptr;             // [n, T] out
    int log_out = 0;                   // write log(product) instead of the product
    void* dst = nullptr;               // instead of acc: rows dst_rows[q] of this
    const int64_t* dst_rows = nullptr; // [*, T] array of the factors' type
    // log_out with lie != null: the log's Hall coordinates through the packed
    // map (sparse_map.cuh) to lie[q * ld_lie + row] instead of the log
    double* lie = nullptr;
    int64_t ld_lie = 0, lie_dim = 0;
    int groups = 0;
    const double* tab = nullptr;
    const uint32_t* goff = nullptr;
    const uint32_t* perm = nullptr;
    const uint32_t* len = nullptr;
    const uint32_t* ent = nullptr;
};

template <int D>
constexpr int chain_first() { return D == 2 ? 3 : D == 3 ? 2 : 1; }

// float64 words of shared memory: a whole row, three times its lower levels
__host__ __device__ constexpr int64_t chain_words(int64_t T, int64_t TL)
{
    return ((T + 3) & ~int64_t(1)) + 3 * ((TL + 3) & ~int64_t(1));
}

// The deepest depth of width D that fits.
template <int D>
constexpr int chain_max_depth()
{
    int64_t words = 0, pw = 1;
    for (int k = 0; k <= kMaxDepth; ++k) {   // words: below level k
        if (chain_words(words + pw, words) * 8 > kChainSmem) return k - 1;
        words += pw;
        pw *= D;
    }
    return kMaxDepth;
}

// lie <- map(xs) by the block's warps, a group of 32 rows at a time; the next
// entries are in flight during the multiply-adds
__device__ __forceinline__ void project_log(const ChainArgs& a, const double* xs, double* lie,
                                            int warp, int nwarps, int lane)
{
    constexpr int kAhead = 8;
    for (int g = warp; g < a.groups; g += nwarps) {
        const uint32_t e0 = __ldg(a.goff + g), longest = (__ldg(a.goff + g + 1) - e0) >> 5;
        const uint32_t row = __ldg(a.perm + g * 32 + lane);
        const uint32_t len = __ldg(a.len + g * 32 + lane);
        uint32_t w[kAhead], wn[kAhead];
        auto entries = [&](uint32_t j, uint32_t (&e)[kAhead]) {
#pragma unroll
            for (int u = 0; u < kAhead; ++u)
                e[u] = j + u < len ? __ldg(a.ent + e0 + lane + (j + u) * 32) : 0u;
        };
        entries(0, w);
        double acc = 0.0;
        for (uint32_t j = 0; j < longest; j += kAhead) {
            entries(j + kAhead, wn);
#pragma unroll
            for (int u = 0; u < kAhead; ++u) {
                if (j + u >= len) break;
                acc = fma(__ldg(a.tab + (w[u] >> 20)), xs[w[u] & 0xfffffu], acc);
            }
#pragma unroll
            for (int u = 0; u < kAhead; ++u) w[u] = wn[u];
        }
        if (row != 0xffffffffu) lie[row] = acc;
    }
}

template <typename TS, int D>
__global__ void __launch_bounds__(kChainThreads, 1)
chain_products_kernel(const ChainArgs a)
{
    constexpr int F = chain_first<D>();
    constexpr int U = Power<D, F>::value;
    constexpr int NMAX = chain_max_depth<D>();
    extern __shared__ __align__(16) unsigned char chain_smem[];
    const int N = a.depth;
    const int TL = (int)a.db[N], T = (int)a.T;
    double* const row_room = reinterpret_cast<double*>(chain_smem);
    double* const low_room = row_room + stage_room(T);
    double* const x_room[2] = {low_room + stage_room(TL), low_room + 2 * stage_room(TL)};
    const int tid = (int)threadIdx.x, B = (int)blockDim.x;
    const int lane = tid & 31, warp = tid >> 5, nwarps = B >> 5;
    const TS* src = static_cast<const TS*>(a.src);

    // Calls unit(level, lane's unit) for the tasks of levels hi down to F that
    // are this warp's, then shorts() for the levels below (one task).
    auto deal = [&](int hi, auto&& unit, auto&& shorts) {
        int t = warp;
        for (int k = max(hi, F - 1); k >= F - 1;) {
            const int tasks = k >= F ? (int)((a.pw[k - F] + 31) >> 5) : 1;
            if (t >= tasks) {
                t -= tasks;
                --k;
                continue;
            }
            if (k < F) {
                shorts();
            } else {
                const uint32_t r = (uint32_t)(t * 32 + lane);
                with_level<F, NMAX>(k, [&](auto kc) { unit(kc, r); });
            }
            t += nwarps;
        }
    };

    for (int64_t q = blockIdx.x; q < a.n; q += gridDim.x) {
        const int64_t o0 = a.stride ? q * a.stride : a.off[q];
        const int64_t o1 = a.stride ? o0 + a.off[q] : a.off[q + 1];
        double* accq = a.acc ? a.acc + q * a.T : nullptr;
        TS* dstq = a.dst ? static_cast<TS*>(a.dst) + a.dst_rows[q] * a.T : nullptr;
        if (o0 == o1 && a.lie) {   // the log of the unit: zero coordinates
            for (int64_t r = tid; r < a.lie_dim; r += B) a.lie[q * a.ld_lie + r] = 0.0;
            continue;
        }
        if (o0 == o1) {   // the unit, or its log
            for (int64_t i = tid; i < a.T; i += B) {
                const double v = (i == 0 && !a.log_out) ? 1.0 : 0.0;
                if (dstq) dstq[i] = (TS)v;
                else accq[i] = v;
            }
            continue;
        }
        // factors' top levels start towards L2 three products ahead
        auto prefetch_top = [&](int64_t r) {
            if (r >= o1) return;
            const char* p = reinterpret_cast<const char*>(src + a.rows[r] * a.T + TL);
            const int64_t bytes = (a.T - TL) * (int64_t)sizeof(TS);
            for (int64_t l = (int64_t)tid * 128; l < bytes; l += (int64_t)B * 128)
                asm volatile("prefetch.global.L2 [%0];" ::"l"(p + l));
        };
        // (before a float32 row is waited for, after a float64 one's copies start)
        if (sizeof(TS) == 4)
            for (int64_t r = o0 + 1; r < o0 + 4; ++r) prefetch_top(r);
        __syncthreads();   // the previous row's reads of the buffers are done
        double* const xs = stage_words(row_room, src + a.rows[o0] * a.T, T, tid, B);
        double* top = xs + TL;
        double* cur = xs;          // lower levels of the running product
        double* nxt = low_room;
        double* fx = nullptr;      // lower levels of the factor
        if (o0 + 1 < o1) fx = stage_words(x_room[0], src + a.rows[o0 + 1] * a.T, TL, tid, B);
        if (sizeof(TS) == 8)
            for (int64_t r = o0 + 1; r < o0 + 4; ++r) prefetch_top(r);
        for (int64_t r = o0 + 1; r < o1; ++r) {
            asm volatile("cp.async.wait_all;" ::: "memory");
            __syncthreads();
            const double* X = fx;
            if (r + 1 < o1)
                fx = stage_words(x_room[(r - o0) & 1], src + a.rows[r + 1] * a.T, TL, tid, B);
            prefetch_top(r + 3);
            const TS* node = src + a.rows[r] * a.T;
            const double node0 = X[0], c0v = cur[0];
            // level k <= N at unit u: base * node0 + splits + c0 * node
            auto unit = [&](auto kc, uint32_t ru) {
                constexpr int K = decltype(kc)::value;
                constexpr int run = Power<D, K - F>::value, begin = LevelStart<D, K>::value;
                if (run % 32 != 0 && ru >= (uint32_t)run) return;
                double acc[U];
                if (K == N) {
                    const TS* np = node + begin + ru;
                    TS nv[U];
#pragma unroll
                    for (int u = 0; u < U; ++u) nv[u] = __ldg(np + u * run);
                    double* tp = xs + begin + ru;
#pragma unroll
                    for (int u = 0; u < U; ++u) acc[u] = tp[u * run] * node0;
                    split_unit<D, F, K, U>(acc, cur, X, ru);
#pragma unroll
                    for (int u = 0; u < U; ++u) tp[u * run] = fma(c0v, (double)nv[u], acc[u]);
                } else {
                    const double* cp = cur + begin + ru;
                    const double* xp = X + begin + ru;
                    double* np = nxt + begin + ru;
#pragma unroll
                    for (int u = 0; u < U; ++u) acc[u] = cp[u * run] * node0;
                    split_unit<D, F, K, U>(acc, cur, X, ru);
#pragma unroll
                    for (int u = 0; u < U; ++u) np[u * run] = fma(c0v, xp[u * run], acc[u]);
                }
            };
            deal(N, unit, [&]() {
                for (int k = 1; k < F && k <= N; ++k)
                    for (int w = lane; w < (int)a.pw[k]; w += 32) {
                        const int o = (int)a.db[k] + w;
                        double v = (k < N ? cur[o] : xs[o]) * node0;
                        int ds = 1;
                        for (int s = 1; s < k; ++s) {
                            ds *= D;
                            v = fma(cur[a.db[k - s] + w / ds], X[a.db[s] + w % ds], v);
                        }
                        v = fma(c0v, k < N ? X[o] : (double)__ldg(node + o), v);
                        if (k < N) nxt[o] = v;
                        else xs[o] = v;
                    }
            });
            if (tid == 0) nxt[0] = c0v * node0;
            double* t = cur;
            cur = nxt;
            nxt = t;
        }
        asm volatile("cp.async.wait_all;" ::: "memory");
        __syncthreads();
        if (a.log_out) {
            // With Y = X - X_0 and R = 0, for deg = N down to 1: R <- (R + c_deg) Y
            // truncated to the levels N - deg + 1 and below, c_deg =
            // (-1)^(deg+1) / deg.  Y's lower levels stay in cur, its top level
            // becomes R's in the last step.
            double* rc = x_room[0];
            double* rn = x_room[1];
            for (int s = 1; s <= N; ++s) {
                const int deg = N - s + 1;
                const double c = a.coeff[deg];
                auto unit = [&](auto kc, uint32_t ru) {
                    constexpr int K = decltype(kc)::value;
                    constexpr int run = Power<D, K - F>::value, begin = LevelStart<D, K>::value;
                    if (run % 32 != 0 && ru >= (uint32_t)run) return;
                    double acc[U];
                    double* to = (K == N ? xs : rn) + begin + ru;
                    const double* from = (K == N ? xs : cur) + begin + ru;
#pragma unroll
                    for (int u = 0; u < U; ++u) acc[u] = c * from[u * run];
                    split_unit<D, F, K, U>(acc, rc, cur, ru);
#pragma unroll
                    for (int u = 0; u < U; ++u) to[u * run] = acc[u];
                };
                deal(s, unit, [&]() {
                    for (int k = 1; k < F && k <= s; ++k)
                        for (int w = lane; w < (int)a.pw[k]; w += 32) {
                            const int o = (int)a.db[k] + w;
                            double v = c * (k < N ? cur[o] : xs[o]);
                            int ds = 1;
                            for (int t = 1; t < k; ++t) {
                                ds *= D;
                                v = fma(rc[a.db[k - t] + w / ds], cur[a.db[t] + w % ds], v);
                            }
                            if (k < N) rn[o] = v;
                            else xs[o] = v;
                        }
                });
                __syncthreads();
                double* t = rc;
                rc = rn;
                rn = t;
            }
            if (tid == 0) rc[0] = 0.0;
            cur = rc;
            __syncthreads();
        }
        if (a.lie) {
            if (cur != xs) {   // the lower levels beside the top
                for (int i = tid; i < TL; i += B) xs[i] = cur[i];
                __syncthreads();
            }
            project_log(a, xs, a.lie + q * a.ld_lie, warp, nwarps, lane);
        } else if (dstq) {
            // straight into the factors' array, rounded once to its type
            for (int i = tid; i < T; i += B) dstq[i] = (TS)(i < TL ? cur[i] : top[i - TL]);
        } else {
            for (int i = tid; i < T; i += B) accq[i] = i < TL ? cur[i] : top[i - TL];
        }
    }
}

using ChainFn = void (*)(ChainArgs);

template <typename TS>
ChainFn chain_fn(int width)
{
    switch (width) {
        case 2: return &chain_products_kernel<TS, 2>;
        case 3: return &chain_products_kernel<TS, 3>;
        case 4: return &chain_products_kernel<TS, 4>;
        case 5: return &chain_products_kernel<TS, 5>;
        case 6: return &chain_products_kernel<TS, 6>;
        case 7: return &chain_products_kernel<TS, 7>;
        case 8: return &chain_products_kernel<TS, 8>;
        default: return nullptr;
    }
}

}  // namespace

bool chain_products_available(const Geometry& g)
{
    return g.width >= 2 && g.width <= 8 && g.depth >= 2 &&
           chain_words(g.size(), g.db[g.depth]) * 8 <= kChainSmem;
}

static int chain_launch(int src_mode, const Geometry& g, int64_t n, double* acc, const void* src,
                        const std::vector<int64_t>& off, const std::vector<int64_t>& src_rows,
                        bool log_out, void* dst, const std::vector<int64_t>* dst_rows,
                        cudaStream_t s, const LieMapsDev* maps = nullptr, double* lie = nullptr,
                        int64_t ld_lie = 0);

int chain_products(int src_mode, const Geometry& g, int64_t n, double* acc, const void* src,
                   const std::vector<int64_t>& off, const std::vector<int64_t>& src_rows,
                   bool log_out, cudaStream_t s)
{
    return chain_launch(src_mode, g, n, acc, src, off, src_rows, log_out, nullptr, nullptr, s);
}

int chain_products_into(int src_mode, const Geometry& g, int64_t n, void* nodes,
                        const std::vector<int64_t>& off, const std::vector<int64_t>& src_rows,
                        const std::vector<int64_t>& dst_rows, cudaStream_t s)
{
    return chain_launch(src_mode, g, n, nullptr, nodes, off, src_rows, false, nodes, &dst_rows, s);
}

bool chain_lie_available(const Geometry& g, const LieMapsDev& maps)
{
    return chain_products_available(g) && maps.t2l.block;
}

int chain_products_lie(int src_mode, const Geometry& g, int64_t n, const void* src,
                       const std::vector<int64_t>& off, const std::vector<int64_t>& src_rows,
                       const LieMapsDev& maps, double* lie, int64_t ld_lie, cudaStream_t s)
{
    if (!chain_lie_available(g, maps)) return fail(RPYB_E_UNSUPPORTED, "no fused projection for this shape");
    return chain_launch(src_mode, g, n, nullptr, src, off, src_rows, true, nullptr, nullptr, s,
                        &maps, lie, ld_lie);
}

static ChainArgs chain_args(const Geometry& g, int64_t n)
{
    ChainArgs a;
    a.T = g.size();
    for (int k = 0; k <= kMaxDepth + 1; ++k) a.db[k] = g.db[k];
    for (int k = 0; k <= kMaxDepth; ++k) a.pw[k] = g.pw[k];
    for (int deg = 1; deg <= g.depth; ++deg) a.coeff[deg] = (deg % 2 == 0 ? -1.0 : 1.0) / deg;
    a.depth = g.depth;
    a.n = n;
    return a;
}

static void set_projection(ChainArgs& a, const LieMapsDev& maps, double* lie, int64_t ld_lie)
{
    const PackedMap& m = maps.t2l;
    a.lie = lie;
    a.ld_lie = ld_lie;
    a.lie_dim = maps.lie_dim;
    a.groups = (int)m.groups;
    a.tab = static_cast<const double*>(m.block);
    a.goff = reinterpret_cast<const uint32_t*>(a.tab + m.ntab);
    a.perm = a.goff + m.groups + 1;
    a.len = a.perm + 32 * m.groups;
    a.ent = a.len + 32 * m.groups;
}

static int run_chain(int src_mode, const Geometry& g, const ChainArgs& a, cudaStream_t s)
{
    const size_t smem = (size_t)chain_words(g.size(), g.db[g.depth]) * 8;
    const int F = g.width == 2 ? 3 : g.width == 3 ? 2 : 1;
    const int64_t threads = row_block_threads(g, g.depth, F, smem, kChainSmem, a.n, kChainThreads);
    const unsigned grid = (unsigned)std::min<int64_t>(a.n, 1 << 20);
    ChainFn fn = src_mode == RPYB_F64 ? chain_fn<double>(g.width) : chain_fn<float>(g.width);
    if (int rc = allow_shared_memory(fn, smem, kChainSmem)) return rc;
    fn<<<grid, (unsigned)threads, smem, s>>>(a);
    RPYB_CUDA(cudaGetLastError());
    return RPYB_OK;
}

int chain_products_lie_strided(int src_mode, const Geometry& g, int64_t n, const void* src,
                               const int64_t* counts, const int64_t* rows, int64_t stride,
                               const LieMapsDev& maps, double* lie, int64_t ld_lie, cudaStream_t s)
{
    if (n == 0) return RPYB_OK;
    if (!chain_lie_available(g, maps)) return fail(RPYB_E_UNSUPPORTED, "no fused projection for this shape");
    ChainArgs a = chain_args(g, n);
    a.off = counts;
    a.rows = rows;
    a.stride = stride;
    a.src = src;
    a.log_out = 1;
    set_projection(a, maps, lie, ld_lie);
    return run_chain(src_mode, g, a, s);
}

static int chain_launch(int src_mode, const Geometry& g, int64_t n, double* acc, const void* src,
                        const std::vector<int64_t>& off, const std::vector<int64_t>& src_rows,
                        bool log_out, void* dst, const std::vector<int64_t>* dst_rows,
                        cudaStream_t s, const LieMapsDev* maps, double* lie, int64_t ld_lie)
{
    if (n == 0) return RPYB_OK;
    if (!chain_products_available(g)) return fail(RPYB_E_UNSUPPORTED, "no chain kernel for this shape");
    if (off[n] == 0 && lie) {
        RPYB_CUDA(cudaMemset2DAsync(lie, (size_t)ld_lie * 8, 0, (size_t)maps->lie_dim * 8,
                                    (size_t)n, s));
        return RPYB_OK;
    }
    if (off[n] == 0 && !dst) {
        if (log_out) {
            RPYB_CUDA(cudaMemsetAsync(acc, 0, (size_t)(n * g.size() * 8), s));
            return RPYB_OK;
        }
        return unit_rows(RPYB_F64, acc, g.size(), g.size(), nullptr, n, s);
    }
    ChainArgs a = chain_args(g, n);
    // offsets and rows in one upload
    std::vector<int64_t> packed(off.begin(), off.begin() + n + 1);
    packed.insert(packed.end(), src_rows.begin(), src_rows.begin() + off[n]);
    if (dst) packed.insert(packed.end(), dst_rows->begin(), dst_rows->begin() + n);
    Scratch sc(nullptr, 0, s);
    void* mem = nullptr;
    int rc;
    if ((rc = sc.get(packed.size() * 8, &mem))) return rc;
    int64_t* d = static_cast<int64_t*>(mem);
    if ((rc = upload_async(d, packed.data(), packed.size() * 8, s))) return rc;
    a.off = d;
    a.rows = d + n + 1;
    a.src = src;
    a.acc = acc;
    a.log_out = log_out ? 1 : 0;
    a.dst = dst;
    a.dst_rows = dst ? d + n + 1 + off[n] : nullptr;
    if (lie) set_projection(a, *maps, lie, ld_lie);
    return run_chain(src_mode, g, a, s);
}

}  // namespace rpyb
