// Batched sparse linear maps with the map packed for warps (sparse_map.cuh).
//
// The Lie <-> tensor maps are a few entries a row with values from a table of
// a dozen numbers.  As CSR with 64-bit indices and float64 values, one thread
// an output word, every batch row read the whole map again (16 bytes an entry,
// uncoalesced across the warp) and gathered its words from L2.  Here an entry
// is 4 bytes, a warp's entry reads are consecutive, and a block computes RB
// batch rows whose words it first copies into shared memory, so an entry read
// feeds RB multiply-adds and a gather costs a shared-memory access.  What
// bounds tensor -> Lie then is those gathers (random columns: 5.3 wavefronts a
// float64 request, L1 80 % busy), Lie -> tensor the stores of y.  Measured on
// B200, 4096 rows at (6,5), CSR with the zero fill of y -> packed: tensor -> Lie
// float64 650 -> 205 us, float32 112 us; Lie -> tensor float64 122 us, float32
// 94 us (HBM time of x and y: 57 and 28 us).
#include <algorithm>
#include <cstring>
#include <new>
#include <numeric>
#include <unordered_map>

#include "sparse_map.cuh"

namespace rpyb {
namespace {

constexpr int kMapThreads = 512;   // most threads a block
// Maps of many entries a row sort their rows by length within windows of this
// many, so that a group's lanes run about equal counts.  Maps of few keep the
// order: their time is in the stores of y, which a sorted group scatters.
// Measured on B200 at (6,5), 4096 float64 rows, in order / sorted: tensor -> Lie
// (15 entries a row) 249 / 210 us, Lie -> tensor (3 entries) 122 / 215 us.
constexpr int64_t kSortWindow = 128;
constexpr int64_t kSortEntries = 8;   // entries a row from which rows are sorted
constexpr uint32_t kColBits = 20;
constexpr int64_t kMaxTab = 4096;
constexpr int64_t kMapRoom = 100 * 1024;   // shared memory of a block when two fit an SM

struct MapArgs {
    const double* tab;
    const uint32_t* goff;
    const uint32_t* perm;
    const uint32_t* len;
    const uint32_t* ent;
    int n_cols, groups, ntab;
    int64_t batch, ld_y, ld_x;
    double scale;
    bool accumulate;
};

template <typename T>
__device__ __forceinline__ void copy_async(T* smem, const T* gmem)
{
    asm volatile("cp.async.ca.shared.global [%0], [%1], %2;" ::"r"(
                     (uint32_t)__cvta_generic_to_shared(smem)),
                 "l"(gmem), "n"(sizeof(T))
                 : "memory");
}

template <typename T, int RB, bool STAGED>
__global__ void __launch_bounds__(kMapThreads)
packed_map_kernel(const MapArgs a, T* __restrict__ y, const T* __restrict__ x)
{
    extern __shared__ __align__(16) unsigned char map_smem[];
    double* tab = reinterpret_cast<double*>(map_smem);
    T* xs = reinterpret_cast<T*>(tab + a.ntab);   // [RB][n_cols] when staged
    const int tid = (int)threadIdx.x;
    const int lane = tid & 31, warp = tid >> 5;
    const int threads = (int)blockDim.x, warps = threads >> 5;
    const int64_t b0 = blockIdx.x * (int64_t)RB;
    for (int i = tid; i < a.ntab; i += threads) tab[i] = __ldg(a.tab + i);
    const T* xr[RB];
#pragma unroll
    for (int r = 0; r < RB; ++r) xr[r] = x + min(b0 + r, a.batch - 1) * a.ld_x;
    if constexpr (STAGED) {
        // all of a thread's words in flight at once
        for (int c = tid; c < a.n_cols; c += threads)
#pragma unroll
            for (int r = 0; r < RB; ++r) copy_async(xs + r * a.n_cols + c, xr[r] + c);
        asm volatile("cp.async.wait_all;" ::: "memory");
    }
    __syncthreads();
    // Heavy groups come first, so a stride of all warps deals them evenly.  A
    // group's row numbers and lengths are read two groups ahead and its first
    // entries one ahead, so that a group does not begin with a chain of three
    // L2 latencies.
    // (more ahead where few rows leave the SM few warps: (2,10) tensor -> Lie, one
    // row of up to 140 entries a word, 12.3 -> 9.6 us)
    constexpr int kAhead = RB == 1 ? 16 : 8;
    const int step = (int)gridDim.y * warps;
    struct Meta {
        uint32_t e0, longest, row, len;
    };
    auto meta = [&](int g) {
        Meta m{0u, 0u, 0xffffffffu, 0u};
        if (g < a.groups) {
            m.e0 = __ldg(a.goff + g);
            m.longest = (__ldg(a.goff + g + 1) - m.e0) >> 5;
            m.row = __ldg(a.perm + g * 32 + lane);
            m.len = __ldg(a.len + g * 32 + lane);
        }
        return m;
    };
    auto entries = [&](const Meta& m, uint32_t j, uint32_t (&w)[kAhead]) {
#pragma unroll
        for (int u = 0; u < kAhead; ++u)
            w[u] = j + u < m.len ? __ldg(a.ent + m.e0 + lane + (j + u) * 32) : 0u;
    };
    int g = blockIdx.y * warps + warp;
    Meta cur = meta(g), next = meta(g + step);
    uint32_t w[kAhead], wn[kAhead];
    entries(cur, 0, w);
    double acc[RB];
#pragma unroll
    for (int r = 0; r < RB; ++r) acc[r] = 0.0;
    for (uint32_t j = 0; g < a.groups;) {
        // the following entries, of this group or the next, are in flight
        // during this chunk's multiply-adds
        const bool done = j + kAhead >= cur.longest;
        if (done) entries(next, 0, wn);
        else entries(cur, j + kAhead, wn);
#pragma unroll
        for (int u = 0; u < kAhead; ++u) {
            if (j + u >= cur.len) break;
            const double v = tab[w[u] >> kColBits];
            const uint32_t c = w[u] & ((1u << kColBits) - 1u);
#pragma unroll
            for (int r = 0; r < RB; ++r) {
                if constexpr (STAGED) acc[r] = fma(v, (double)xs[r * a.n_cols + c], acc[r]);
                else acc[r] = fma(v, (double)__ldg(xr[r] + c), acc[r]);
            }
        }
#pragma unroll
        for (int u = 0; u < kAhead; ++u) w[u] = wn[u];
        j += kAhead;
        if (!done) continue;
        if (cur.row != 0xffffffffu) {
#pragma unroll
            for (int r = 0; r < RB; ++r) {
                if (b0 + r >= a.batch) break;
                T* yp = y + (b0 + r) * a.ld_y + cur.row;
                *yp = a.accumulate ? (T)((double)*yp + a.scale * acc[r]) : (T)(a.scale * acc[r]);
            }
        }
#pragma unroll
        for (int r = 0; r < RB; ++r) acc[r] = 0.0;
        j = 0;
        g += step;
        cur = next;
        next = meta(g + step);
    }
}

template <typename T, int RB, bool STAGED>
int launch_map(const MapArgs& a, T* y, const T* x, cudaStream_t s)
{
    auto fn = packed_map_kernel<T, RB, STAGED>;
    const size_t smem = (size_t)a.ntab * 8 + (STAGED ? (size_t)RB * a.n_cols * sizeof(T) : 0);
    if (int rc = allow_shared_memory(fn, smem, 2 * kMapRoom)) return rc;
    const int64_t blocks = (a.batch + RB - 1) / RB;
    if (blocks > 0x7fffffff) return fail(RPYB_E_UNSUPPORTED, "batch too large");
    // few rows: blocks share a row block's groups
    const int64_t split = std::max<int64_t>(
        1, std::min<int64_t>(296 / blocks, (a.groups + kMapThreads / 32 - 1) / (kMapThreads / 32)));
    // a warp a group of a small map (two at least, to copy the rows): 16 warps
    // for one group of (2,3), 30000 float64 rows, took 21 us, two take 6.0
    const int threads = (int)std::max<int64_t>(64, std::min<int64_t>(kMapThreads, 32 * (int64_t)a.groups));
    fn<<<dim3((unsigned)blocks, (unsigned)split), threads, smem, s>>>(a, y, x);
    RPYB_CUDA(cudaGetLastError());
    return RPYB_OK;
}

template <typename T>
int launch_map_rows(const MapArgs& a, T* y, const T* x, cudaStream_t s)
{
    // As many rows a block as leave room for two blocks an SM and blocks for
    // every SM; a row that fits only alone is staged alone, a longer one read
    // where it is.
    const int64_t row = (int64_t)a.n_cols * sizeof(T), room = kMapRoom - a.ntab * 8;
    const int64_t want = std::max<int64_t>(1, a.batch / 296);
    if (8 * row <= room && want >= 8) return launch_map<T, 8, true>(a, y, x, s);
    if (4 * row <= room && want >= 4) return launch_map<T, 4, true>(a, y, x, s);
    if (2 * row <= room && want >= 2) return launch_map<T, 2, true>(a, y, x, s);
    if (row <= 2 * room) return launch_map<T, 1, true>(a, y, x, s);
    return launch_map<T, 2, false>(a, y, x, s);
}

}  // namespace

// Where the rows of a map go: its groups' rows and longest counts, heaviest
// group first.
struct PackLayout {
    std::vector<uint32_t> count;     // entries kept, per row
    std::vector<int64_t> order;      // rows, 32 to a group
    std::vector<uint32_t> longest;   // per group of `order`
    std::vector<int64_t> by_len;     // groups, longest first
    int64_t entries = 0, slots = 0;
};

static bool pack_layout(int64_t n_rows, int64_t n_cols, const int64_t* ptr, const int64_t* idx,
                        PackLayout& l)
{
    if (n_cols > (int64_t(1) << kColBits) || n_rows >= 0x7fffffff) return false;
    l.count.assign(n_rows, 0);
    for (int64_t r = 0; r < n_rows; ++r) {
        uint32_t c = 0;
        for (int64_t k = ptr[r]; k < ptr[r + 1]; ++k) c += (uint64_t)idx[k] < (uint64_t)n_cols;
        l.count[r] = c;
        l.entries += c;
    }
    l.order.resize(n_rows);
    std::iota(l.order.begin(), l.order.end(), int64_t(0));
    for (int64_t r0 = 0; l.entries >= kSortEntries * n_rows && r0 < n_rows; r0 += kSortWindow)
        std::stable_sort(l.order.begin() + r0, l.order.begin() + std::min(r0 + kSortWindow, n_rows),
                         [&](int64_t p, int64_t q) { return l.count[p] > l.count[q]; });
    const int64_t groups = (n_rows + 31) / 32;
    l.longest.assign(groups, 0);
    for (int64_t g = 0; g < groups; ++g)
        for (int64_t i = g * 32; i < std::min(g * 32 + 32, n_rows); ++i)
            l.longest[g] = std::max(l.longest[g], l.count[l.order[i]]);
    l.by_len.resize(groups);
    std::iota(l.by_len.begin(), l.by_len.end(), int64_t(0));
    std::stable_sort(l.by_len.begin(), l.by_len.end(),
                     [&](int64_t p, int64_t q) { return l.longest[p] > l.longest[q]; });
    for (int64_t g = 0; g < groups; ++g) l.slots += 32 * (int64_t)l.longest[g];
    return l.slots < (int64_t(1) << 32);
}

// Value ids by the values' bits, through a direct-mapped cache: the maps have a
// dozen values in no predictable order.
class ValueTable {
public:
    std::vector<double> tab;
    // false when there are too many
    bool id(double v, uint32_t* out)
    {
        uint64_t bits;
        std::memcpy(&bits, &v, sizeof bits);
        Slot& s = cache_[(bits * 0x9E3779B97F4A7C15ull) >> 56];
        if (s.id == kNone || s.bits != bits) {
            auto it = ids_.find(bits);
            if (it == ids_.end()) {
                if ((int64_t)tab.size() == kMaxTab) return false;
                it = ids_.emplace(bits, (uint32_t)tab.size()).first;
                tab.push_back(v);
            }
            s = Slot{bits, it->second};
        }
        *out = s.id;
        return true;
    }

private:
    static constexpr uint32_t kNone = 0xffffffffu;
    struct Slot {
        uint64_t bits = 0;
        uint32_t id = kNone;
    };
    Slot cache_[256];
    std::unordered_map<uint64_t, uint32_t> ids_;
};

bool pack_map(int64_t n_rows, int64_t n_cols, const int64_t* ptr, const int64_t* idx,
              const double* val, PackedMap& m, std::vector<unsigned char>& block)
{
    m = PackedMap{};
    m.n_rows = n_rows;
    m.n_cols = n_cols;
    PackLayout l;
    if (!pack_layout(n_rows, n_cols, ptr, idx, l)) return false;
    // the entries first: the number of distinct values decides where they go
    std::vector<uint32_t> ent(l.slots, 0);
    ValueTable values;
    m.groups = (int64_t)l.longest.size();
    m.slots = l.slots;
    uint32_t e0 = 0;
    for (int64_t i = 0; i < m.groups; ++i) {
        const int64_t g = l.by_len[i];
        for (int lane = 0; lane < 32 && g * 32 + lane < n_rows; ++lane) {
            const int64_t r = l.order[g * 32 + lane];
            uint32_t* e = ent.data() + e0 + lane;
            for (int64_t k = ptr[r]; k < ptr[r + 1]; ++k) {
                if ((uint64_t)idx[k] >= (uint64_t)n_cols) continue;
                uint32_t vid;
                if (!values.id(val[k], &vid)) return false;
                *e = (uint32_t)idx[k] | (vid << kColBits);
                e += 32;
            }
        }
        e0 += 32 * l.longest[g];
    }
    m.ntab = (int64_t)values.tab.size();
    block.resize(packed_map_bytes(m));
    double* btab = reinterpret_cast<double*>(block.data());
    std::copy(values.tab.begin(), values.tab.end(), btab);
    uint32_t* goff = reinterpret_cast<uint32_t*>(btab + m.ntab);
    uint32_t* perm = goff + m.groups + 1;
    uint32_t* len = perm + 32 * m.groups;
    goff[0] = 0;
    for (int64_t i = 0; i < m.groups; ++i) {
        const int64_t g = l.by_len[i];
        goff[i + 1] = goff[i] + 32 * l.longest[g];
        for (int lane = 0; lane < 32; ++lane) {
            const bool has = g * 32 + lane < n_rows;
            const int64_t r = has ? l.order[g * 32 + lane] : 0;
            perm[i * 32 + lane] = has ? (uint32_t)r : 0xffffffffu;
            len[i * 32 + lane] = has ? l.count[r] : 0u;
        }
    }
    std::memcpy(len + 32 * m.groups, ent.data(), ent.size() * sizeof(uint32_t));
    return true;
}

int launch_packed_map(int dtype, const PackedMap& m, int64_t batch, void* y, int64_t ld_y,
                      const void* x, int64_t ld_x, double scale, bool accumulate, cudaStream_t s)
{
    if (batch <= 0 || m.n_rows <= 0) return RPYB_OK;
    MapArgs a{};
    a.tab = static_cast<const double*>(m.block);
    a.goff = reinterpret_cast<const uint32_t*>(a.tab + m.ntab);
    a.perm = a.goff + m.groups + 1;
    a.len = a.perm + 32 * m.groups;
    a.ent = a.len + 32 * m.groups;
    a.n_cols = (int)m.n_cols;
    a.groups = (int)m.groups;
    a.ntab = (int)m.ntab;
    a.batch = batch;
    a.ld_y = ld_y;
    a.ld_x = ld_x;
    a.scale = scale;
    a.accumulate = accumulate;
    if (dtype == RPYB_F64)
        return launch_map_rows(a, static_cast<double*>(y), static_cast<const double*>(x), s);
    return launch_map_rows(a, static_cast<float*>(y), static_cast<const float*>(x), s);
}

}  // namespace rpyb

using namespace rpyb;

extern "C" {

RPYB_API int64_t rpyb_sparse_pack(int64_t n_rows, int64_t n_cols, const int64_t* indptr,
                                  const int64_t* indices, const double* values, void* block,
                                  int64_t block_bytes, int64_t* layout)
{
    if (n_rows < 0 || n_cols < 0) return fail(RPYB_E_INVALID, "negative size");
    if (!indptr || !layout) return fail(RPYB_E_INVALID, "null pointer");
    // a row that ends before it begins is empty, as in rpyb_sparse_map
    for (int64_t r = 0; r < n_rows; ++r)
        if (indptr[r + 1] > indptr[r] && (!indices || !values))
            return fail(RPYB_E_INVALID, "null pointer");
    PackedMap m;
    try {
        if (!block) {
            // room for the block whatever its number of distinct values
            PackLayout l;
            if (!pack_layout(n_rows, n_cols, indptr, indices, l))
                return fail(RPYB_E_UNSUPPORTED, "map too large to pack");
            m.groups = (int64_t)l.longest.size();
            m.slots = l.slots;
            m.ntab = std::min(l.entries, kMaxTab);
            return (int64_t)packed_map_bytes(m);
        }
        std::vector<unsigned char> packed;
        if (!pack_map(n_rows, n_cols, indptr, indices, values, m, packed))
            return fail(RPYB_E_UNSUPPORTED, "map too large or with too many distinct values to pack");
        if (block_bytes < (int64_t)packed.size()) return fail(RPYB_E_INVALID, "block too small");
        std::memcpy(block, packed.data(), packed.size());
        layout[0] = m.groups;
        layout[1] = m.slots;
        layout[2] = m.ntab;
        return (int64_t)packed.size();
    } catch (const std::bad_alloc&) {
        return fail(RPYB_E_NOMEM, "out of host memory");
    }
}

RPYB_API int rpyb_sparse_map_packed(int dtype, int64_t n_rows, int64_t n_cols, int64_t batch,
                                    const void* block, const int64_t* layout, void* y,
                                    const void* x, int64_t ld_y, int64_t ld_x, double scale,
                                    int accumulate, void* stream)
{
    if (dtype != RPYB_F32 && dtype != RPYB_F64) return fail(RPYB_E_INVALID, "unsupported dtype");
    if (n_rows < 0 || n_cols < 0 || batch < 0) return fail(RPYB_E_INVALID, "negative size");
    if (batch == 0 || n_rows == 0) return RPYB_OK;
    if (!block || !layout || !y || !x) return fail(RPYB_E_INVALID, "null pointer");
    if (batch > 1 && (ld_y < n_rows || ld_x < n_cols))
        return fail(RPYB_E_INVALID, "row stride smaller than the vector size");
    PackedMap m;
    m.n_rows = n_rows;
    m.n_cols = n_cols;
    m.groups = layout[0];
    m.slots = layout[1];
    m.ntab = layout[2];
    m.block = block;
    if (m.groups != (n_rows + 31) / 32 || m.slots < 0 || m.ntab < 0 || m.ntab > kMaxTab ||
        n_cols > (int64_t(1) << kColBits))
        return fail(RPYB_E_INVALID, "inconsistent packed layout");
    return launch_packed_map(dtype, m, batch, y, ld_y, x, ld_x, scale, accumulate != 0,
                             static_cast<cudaStream_t>(stream));
}

}  // extern "C"
