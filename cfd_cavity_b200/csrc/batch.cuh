// batch.cuh -- many cavities of uneven size and Rayleigh number advanced by
// one launch per lattice step.
//
// Each cavity is an ordinary Impl<St> (own buffers, REF/PC state machine,
// diagnostics); the batch only replaces their per-cavity fused launches by
// one persistent-grid kernel over a work list of (cavity, 32-column x
// `rows`-row) tiles: grid = ctas_per_sm x #SMs CTAs of 128 threads that
// stride over the list.  Tiles are ordered cavity-major, row-block-minor, so
// the tiles in flight at one time are neighbours and the halo rows they
// share are served by L2.  Where that pays (ungrouped_steps), a call's steps run
// group of cavities by group (setup_groups), so that a group's state stays in the
// L2 between its steps.  Per-cavity step scalars (ramps, seeds, wall temperature
// pointers) come from a device table precomputed on the host with
// the single-cavity code (Impl::scalars), row min(step, spin_up), and every
// node runs the same fused_node() as k_fused: a cavity advanced in a batch
// is bit-identical to the same cavity advanced alone.  Steps run as CUDA
// graphs of GRAPH_STEPS launches reading a device step counter.
#pragma once

#include "partition.h"
#include "solver.cuh"
#include "tile.cuh"
#include "tilex.cuh"
#include "xpair.cuh"

#include <limits>

namespace cav {

template <class St>
struct BatchCav {
    St* pop[2];
    typename Fmt<St>::A* fy;
    typename Fmt<St>::A* nut;
    Geom G;
    int parity;   // buffer holding the state at batch step s: pop[(parity + s) & 1]
    int spin_up;  // scalar-table row of the steady state
};

struct BatchItem {
    int cav, tx0, ty0, rows;
};

// A work item with its cavity beside it, for the one-CTA-per-item kernels: a CTA
// reads it and its scalars' row, and nothing else stands before its population
// loads (with the cavity looked up by the item's index, and the row by the
// cavity's spin-up, three loads in a row did: B200, 64 cavities, us per step f16sr
// 40.0 / 38.9 and FP32 48.1 / 45.7 with k_batch_x, bfloat16 37.3 / 36.1, its
// stochastic form 39.8 / 41.0).
template <class St>
struct BatchWork {
    BatchCav<St> cv;
    BatchItem item;
};

constexpr int BATCH_THREADS = 128;

// The scalar table's row of step s: row r holds every cavity's scalars of step
// min(r, its spin-up), the last one (n_rows - 1 = the longest spin-up) the
// steady state of all.
__device__ __forceinline__ long long scalar_row(long long s, int n_rows) { return s < n_rows - 1 ? s : n_rows - 1; }
template <class St, bool WRITE_NUT>
__global__ void __launch_bounds__(BATCH_THREADS)
    k_batch(const BatchCav<St>* __restrict__ cavs, const BatchItem* __restrict__ items, int n_items,
            const StepScalars<typename Fmt<St>::A>* __restrict__ table, int n_cav, long long step,
            const long long* __restrict__ step_dev) {
    using A = typename Fmt<St>::A;
    const long long s = step_dev ? *step_dev + step : step;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    for (int it = blockIdx.x; it < n_items; it += gridDim.x) {
        const BatchItem item = items[it];
        const BatchCav<St> cv = cavs[item.cav];
        const Geom G = cv.G;
        const int row = s < cv.spin_up ? int(s) : cv.spin_up;
        StepScalars<A> c = table[(long long)row * n_cav + item.cav];
        c.step = s;
        c.step_dev = nullptr;
        const int cur = (cv.parity + int(s & 1)) & 1;
        const St* src = cv.pop[cur];
        St* dst = cv.pop[cur ^ 1];
        const int ix = item.tx0 + lane;
        if (ix < G.nx) {
            for (int r = w; r < item.rows; r += BATCH_THREADS / 32)
                fused_node<St, WRITE_NUT, false, false>(src, dst, cv.fy, cv.nut, nullptr, nullptr, G, ix,
                                                        item.ty0 + r, c);
        }
    }
}

// The same node body with one CTA per (cavity, 32-column x rows) item, one
// node per thread (no persistent loop): the per-cavity pointers and scalars
// are not kept live across items, so the kernel needs the registers of
// k_fused, not of k_batch; capped at 56 (with 128-thread CTAs, 9 resident
// per SM; a word or three spilled to L1; on a B200 +3 % binary16, +15 %
// bfloat16 with stochastic rounding against 64 registers and 8 CTAs).  FP64's
// node needs 154 and spills at 56: 128 there (64 cavities: 370 us at 56, 142 at 128).
template <class St, bool WRITE_NUT>
__global__ void __maxnreg__((std::is_same<St, double>::value ? 128 : 56))
    k_batch_np(const BatchWork<St>* __restrict__ work, const StepScalars<typename Fmt<St>::A>* __restrict__ table,
               int n_rows, int n_cav, long long step, const long long* __restrict__ step_dev) {
    using A = typename Fmt<St>::A;
    pdl_wait();
    const long long s = step_dev ? *step_dev + step : step;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const BatchWork<St>& wk = work[blockIdx.x];
    const BatchItem item = wk.item;
    StepScalars<A> c = table[scalar_row(s, n_rows) * n_cav + item.cav];
    c.step = s;
    c.step_dev = nullptr;
    St *const p0 = wk.cv.pop[0], *const p1 = wk.cv.pop[1];
    const bool cur = (wk.cv.parity + int(s & 1)) & 1;
    const int ix = item.tx0 + lane;
    if (ix < wk.cv.G.nx && w < item.rows)
        fused_node<St, WRITE_NUT, false, false>(cur ? p1 : p0, cur ? p0 : p1, wk.cv.fy, wk.cv.nut, nullptr, nullptr,
                                                wk.cv.G, ix, item.ty0 + w, c);
}

// k_batch_np with two rows per thread (fused_pair: the arithmetic of both
// nodes on packed FP32x2 lanes): rows / 2 warps per item.  FP32-arithmetic
// formats only.  Register budget 96 (10 resident 64-thread CTAs per SM, a
// few words spilled to L1): more warps to hide the loads' latency beat the
// spill traffic on a B200.
template <class St, bool WRITE_NUT>
__global__ void __maxnreg__(96)
    k_batch_np2(const BatchWork<St>* __restrict__ work, const StepScalars<float>* __restrict__ table, int n_rows,
                int n_cav, long long step, const long long* __restrict__ step_dev) {
    pdl_wait();
    const long long s = step_dev ? *step_dev + step : step;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const BatchWork<St>& wk = work[blockIdx.x];
    const BatchItem item = wk.item;
    StepScalars<float> c = table[scalar_row(s, n_rows) * n_cav + item.cav];
    c.step = s;
    c.step_dev = nullptr;
    St *const p0 = wk.cv.pop[0], *const p1 = wk.cv.pop[1];
    const bool cur = (wk.cv.parity + int(s & 1)) & 1;
    const int ix = item.tx0 + lane;
    if (ix < wk.cv.G.nx && 2 * w < item.rows)
        fused_pair<St, WRITE_NUT, false>(cur ? p1 : p0, cur ? p0 : p1, wk.cv.fy, wk.cv.nut, nullptr, nullptr, wk.cv.G,
                                         ix, item.ty0 + 2 * w, 2 * w + 1 < item.rows, c);
}

// The node-pair body of k_fused_x (xpair.cuh: two x-adjacent nodes per
// thread, every plane one 32-bit word or float2) with one CTA per (cavity,
// 64-column x rows) item: warp w takes row ty0 + w.
template <class St, bool WRITE_NUT>
__global__ void __maxnreg__(XPAIR_MAXNREG)
    k_batch_x(const BatchWork<St>* __restrict__ work, const StepScalars<float>* __restrict__ table, int n_rows,
              int n_cav, long long step, const long long* __restrict__ step_dev) {
    pdl_wait();
    const long long s = step_dev ? *step_dev + step : step;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const BatchWork<St>& wk = work[blockIdx.x];
    const BatchItem item = wk.item;
    StepScalars<float> c = table[scalar_row(s, n_rows) * n_cav + item.cav];
    c.step = s;
    c.step_dev = nullptr;
    St *const p0 = wk.cv.pop[0], *const p1 = wk.cv.pop[1];
    const bool cur = (wk.cv.parity + int(s & 1)) & 1;
    const int ix = item.tx0 + 2 * lane;
    if (ix < wk.cv.G.nx && w < item.rows)
        fused_xpair<St, WRITE_NUT, false>(cur ? p1 : p0, cur ? p0 : p1, wk.cv.fy, wk.cv.fy, wk.cv.nut, nullptr, nullptr,
                                          wk.cv.G, ix, item.ty0 + w, c);
}

// Which kernel runs a batched step, and the parameters it uses:
//   0  k_batch      persistent grid of ctas_per_sm x #SMs CTAs over
//                   32-column x rows_per_item tiles, one thread per node;
//   1, 2  k_tile    TMA-staged shared-memory tiles of shape 1 or 2,
//                   ctas_per_sm persistent CTAs per SM;
//   3  k_batch_np   one CTA per 32-column x rows_per_item item (rows_per_item
//                   in {1, 2, 4, 8}), one node per thread;
//   4  k_batch_np2  the same items, two rows per thread on packed FP32x2
//                   lanes (rows_per_item in {2, 4, 8}; FP32-arithmetic formats);
//   5  k_batch_x    one CTA per 64-column x rows_per_item item (rows_per_item
//                   in {1, 2, 4, 8}), two x-adjacent nodes per thread, every
//                   plane one 32-bit word (FP32: one float2; not FP64);
//   6  k_tile_x     the node-pair body on TMA-staged shared-memory tiles of
//                   64 columns x rows_per_item rows (4 or 8), ctas_per_sm
//                   persistent CTAs per SM (16-bit formats).
// A kernel a format has no version of runs as kernel 3 (FP64: 4, 5 and 6;
// FP32: 6).  Parameters a kernel does not use are ignored.
struct BatchTuning {
    int rows_per_item = 4;
    int ctas_per_sm = 8;
    int kernel = 3;
};

struct BatchBase {
    virtual ~BatchBase() = default;
    virtual void setup() = 0;
    virtual void step(int64_t n) = 0;
    virtual void set_tuning(const BatchTuning& t) = 0;
    virtual double time_steps(int steps) = 0;  // ms for `steps` batched steps (advances the state)
    virtual void sync() = 0;
    virtual void set_stall_copies(bool on) = 0;
    std::vector<Solver*> cavs;  // owned
    BatchTuning tun;
    cudaStream_t stream = nullptr;
    int64_t time_step = 0;
    int64_t launches = 0;
    long long total_nodes = 0;
    std::string err;
};

template <class St>
struct Batch final : BatchBase {
    using A = typename Fmt<St>::A;
    std::vector<Impl<St>*> cv;
    BatchCav<St>* d_cavs = nullptr;
    BatchItem* d_items = nullptr;     // the items of kernel 0
    BatchWork<St>* d_work = nullptr;  // the items of kernels 3, 4 and 5 with their cavities
    std::vector<BatchItem> items;     // the current kernel's work list
    std::vector<BatchCav<St>> hcavs;  // host copy of d_cavs
    bool work_dirty = true;
    StepScalars<A>* d_table = nullptr;
    long long* step_dev = nullptr;
    long long step_dev_val = -1;
    int n_sm = 0, table_rows = 0;
    // Cavities [c0, c1) that are stepped together, their items in the work
    // list of the current kernel, and GRAPH_STEPS of their steps as a graph
    // (see setup_groups).
    struct Group {
        int c0, c1, item0 = 0, n_items = 0;
        cudaGraphExec_t graph = nullptr;
    };
    std::vector<Group> groups;
    Group every{0, 0};  // all cavities at once (calls that are too short for groups)
    bool cavs_dirty = true;
    // the tile kernel (tile.cuh)
    TileCav<St>* d_tcavs = nullptr;
    CUtensorMap* d_maps[3] = {nullptr, nullptr, nullptr};   // per tile shape
    // the node-pair tile kernel: tensor maps and tile lists per tile height (4, 8)
    CUtensorMap* d_xmaps[2] = {nullptr, nullptr};
    CUtensorMap* d_fmaps[2] = {nullptr, nullptr};  // the Guo force field of every cavity
    TileItem* d_xitems[2] = {nullptr, nullptr};
    std::vector<int> xitem0[2];                             // first tile of every cavity, then their number
    int occ = 0;                                            // resident CTAs per SM of the tile kernel in use
    TileItem* d_titems[3] = {nullptr, nullptr, nullptr};
    unsigned* d_err = nullptr;
    unsigned* h_err = nullptr;  // pinned copy of *d_err
    std::vector<int> titem0[3];
    bool stall_copies = false;  // test of the bounded waits: arm the barriers, issue no copy

    ~Batch() override {
        drop_graphs();
        if (h_err) cudaFreeHost(h_err);
        void* bufs[] = {d_cavs,      d_items, d_work,     d_table, step_dev, d_tcavs,   d_maps[1],
                        d_maps[2],   d_titems[1], d_titems[2], d_err,  d_xmaps[0],
                        d_xmaps[1],  d_xitems[0], d_xitems[1], d_fmaps[0], d_fmaps[1]};
        for (void* b : bufs)
            if (b) cudaFree(b);
        for (Solver* s : cavs) delete s;
        if (stream) cudaStreamDestroy(stream);
    }

    // Builds the device tables once all cavities exist (sharing `stream`).
    void setup() override {
        for (Solver* s : cavs) cv.push_back(static_cast<Impl<St>*>(s));
        int dev = 0;
        CK(cudaGetDevice(&dev));
        CK(cudaDeviceGetAttribute(&n_sm, cudaDevAttrMultiProcessorCount, dev));
        const int n = int(cv.size());
        int max_spin = 0;
        for (auto* c : cv) {
            max_spin = std::max<int>(max_spin, int(c->spin_up));
            total_nodes += (long long)c->p.nx * c->p.ny;
        }
        table_rows = max_spin + 1;
        std::vector<StepScalars<A>> tab(size_t(table_rows) * n);
        for (int r = 0; r < table_rows; ++r)
            for (int i = 0; i < n; ++i) tab[size_t(r) * n + i] = cv[i]->scalars(std::min<int64_t>(r, cv[i]->spin_up));
        CK(cudaMalloc(&d_table, sizeof(StepScalars<A>) * tab.size()));
        CK(cudaMemcpyAsync(d_table, tab.data(), sizeof(StepScalars<A>) * tab.size(), cudaMemcpyHostToDevice,
                           stream));
        CK(cudaMalloc(&d_cavs, sizeof(BatchCav<St>) * n));
        CK(cudaMalloc(&step_dev, sizeof(long long)));
        CK(cudaMalloc(&d_tcavs, sizeof(TileCav<St>) * n));
        CK(cudaMalloc(&d_err, sizeof(unsigned)));
        CK(cudaMemsetAsync(d_err, 0, sizeof(unsigned), stream));
        CK(cudaMallocHost(&h_err, sizeof(unsigned)));
        *h_err = 0;
        setup_groups();
        setup_tiles<1>();
        setup_tiles<2>();
        if constexpr (is_p16<St>::value) {
            setup_xtiles<4>(0);
            setup_xtiles<8>(1);
        }
        set_tuning(tun);
        CK(cudaStreamSynchronize(stream));
    }

    // The cavities are independent, so a call's steps are run for one group of
    // them after another, cut so that a group's state stays in the L2 from step to
    // step where the cavities' sizes allow it (partition.h).
    void setup_groups() {
        int l2 = 0;
        CK(cudaDeviceGetAttribute(&l2, cudaDevAttrL2CacheSize, cv[0]->p.device));
        std::vector<size_t> bytes;
        for (auto* c : cv) bytes.push_back(c->field_elems() * (2 * NPLANES * sizeof(St) + sizeof(A)));
        const std::vector<int> first = partition_groups(bytes, size_t(l2));
        for (size_t i = 0; i + 1 < first.size(); ++i) groups.push_back(Group{first[i], first[i + 1]});
        every.c1 = first.back();
    }

    // First item of every cavity (and the number of items) in a cavity-major list.
    template <class Item>
    std::vector<int> first_items(const std::vector<Item>& items) const {
        std::vector<int> f(cv.size() + 1, 0);
        for (const Item& it : items) ++f[it.cav + 1];
        for (size_t i = 0; i < cv.size(); ++i) f[i + 1] += f[i];
        return f;
    }

    // Tensor maps of both population buffers of every cavity and the tile
    // list, for tile shape V.
    template <int V>
    void setup_tiles() {
        const int n = int(cv.size());
        std::vector<CUtensorMap> maps(2 * size_t(n));
        for (int i = 0; i < n; ++i)
            for (int b = 0; b < 2; ++b) maps[2 * size_t(i) + b] = make_tile_map<St, V>(cv[i]->pop[b], cv[i]->G);
        CK(cudaMalloc(&d_maps[V], sizeof(CUtensorMap) * maps.size()));
        CK(cudaMemcpyAsync(d_maps[V], maps.data(), sizeof(CUtensorMap) * maps.size(), cudaMemcpyHostToDevice,
                           stream));
        std::vector<std::pair<int, int>> sizes;
        for (auto* c : cv) sizes.push_back({c->p.nx, c->p.ny});
        std::vector<TileItem> ti;
        tile_items(sizes, TileShape<St, V>::TY, ti);
        titem0[V] = first_items(ti);
        CK(cudaMalloc(&d_titems[V], sizeof(TileItem) * ti.size()));
        CK(cudaMemcpyAsync(d_titems[V], ti.data(), sizeof(TileItem) * ti.size(), cudaMemcpyHostToDevice, stream));
        CK(cudaFuncSetAttribute(k_tile<St, V, false, false>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                TileShape<St, V>::SMEM));
        CK(cudaFuncSetAttribute(k_tile<St, V, true, false>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                TileShape<St, V>::SMEM));
        CK(cudaStreamSynchronize(stream));
    }

    // Tensor maps (64 + 16 columns x TY + 4 rows x 18 planes) and the tile
    // list of the node-pair tile kernel for tile height TY.
    template <int TY>
    void setup_xtiles(int slot) {
        using TS = TileXShape<TY>;
        const int n = int(cv.size());
        std::vector<CUtensorMap> maps(2 * size_t(n));
        for (int i = 0; i < n; ++i)
            for (int b = 0; b < 2; ++b) maps[2 * size_t(i) + b] = make_box_map<St>(cv[i]->pop[b], cv[i]->G, TX_BX, TS::BY);
        CK(cudaMalloc(&d_xmaps[slot], sizeof(CUtensorMap) * maps.size()));
        CK(cudaMemcpyAsync(d_xmaps[slot], maps.data(), sizeof(CUtensorMap) * maps.size(), cudaMemcpyHostToDevice,
                           stream));
        std::vector<CUtensorMap> fmaps(n);
        if constexpr (is_p16<St>::value)
            for (int i = 0; i < n; ++i) fmaps[i] = make_field_map(cv[i]->fy, cv[i]->G, TX_W, TY);
        CK(cudaMalloc(&d_fmaps[slot], sizeof(CUtensorMap) * fmaps.size()));
        CK(cudaMemcpyAsync(d_fmaps[slot], fmaps.data(), sizeof(CUtensorMap) * fmaps.size(), cudaMemcpyHostToDevice,
                           stream));
        std::vector<std::pair<int, int>> sizes;
        for (auto* c : cv) sizes.push_back({c->p.nx, c->p.ny});
        std::vector<TileItem> ti;
        tilex_items(sizes, TY, ti);
        xitem0[slot] = first_items(ti);
        CK(cudaMalloc(&d_xitems[slot], sizeof(TileItem) * ti.size()));
        CK(cudaMemcpyAsync(d_xitems[slot], ti.data(), sizeof(TileItem) * ti.size(), cudaMemcpyHostToDevice, stream));
        if constexpr (is_p16<St>::value) {
            CK(cudaFuncSetAttribute(k_tile_x<St, TY, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, TS::SMEM));
            CK(cudaFuncSetAttribute(k_tile_x<St, TY, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, TS::SMEM));
        }
        CK(cudaStreamSynchronize(stream));
    }

    template <int TY>
    int xtile_occ() {
        int n = 1;
        if constexpr (is_p16<St>::value)
            CK(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, k_tile_x<St, TY, false>, TileXShape<TY>::THREADS,
                                                             TileXShape<TY>::SMEM));
        return n;
    }

    template <int V>
    int tile_occ() {
        int n = 1;
        CK(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, k_tile<St, V, false, false>, TileShape<St, V>::THREADS,
                                                         TileShape<St, V>::SMEM));
        return n;
    }

    // Persistent CTAs over n work items.
    int grid_of(int n) const { return std::max(1, std::min(n, std::max(1, std::min(tun.ctas_per_sm, occ)) * n_sm)); }

    // The kernel this format runs for a requested one (see BatchTuning).
    static int effective_kernel(int k) {
        if (k == 5 && !has_pairs<St>::value) k = 3;
        if (k == 6 && !is_p16<St>::value) k = 3;
        if (k == 4 && !Fmt<St>::SHIFT) k = 3;
        return k;
    }

    void set_tuning(const BatchTuning& t) override {
        if (t.rows_per_item < 1 || t.rows_per_item > 1024 || t.ctas_per_sm < 1 || t.ctas_per_sm > 32 ||
            t.kernel < 0 || t.kernel > 6)
            throw ArgError{CAV_ERR_ARG, "tuning out of range"};
        const int k = effective_kernel(t.kernel);
        const int r = t.rows_per_item;
        if ((k == 3 || k == 5) && !(r == 1 || r == 2 || r == 4 || r == 8))
            throw ArgError{CAV_ERR_ARG, "rows_per_item of kernels 3 and 5 must be 1, 2, 4 or 8"};
        if (k == 4 && !(r == 2 || r == 4 || r == 8))
            throw ArgError{CAV_ERR_ARG, "rows_per_item of kernel 4 must be 2, 4 or 8"};
        if (k == 6 && !(r == 4 || r == 8)) throw ArgError{CAV_ERR_ARG, "rows_per_item of kernel 6 must be 4 or 8"};
        tun = t;
        // work items: 64 columns for the node-pair kernel, 32 otherwise
        const int width = k == 5 ? 64 : 32;
        items.clear();
        for (int i = 0; i < int(cv.size()); ++i) {
            const int nx = cv[i]->p.nx, ny = cv[i]->p.ny;
            for (int y0 = 0; y0 < ny; y0 += r)
                for (int x0 = 0; x0 < nx; x0 += width) items.push_back({i, x0, y0, std::min(r, ny - y0)});
        }
        if (d_items) CK(cudaFree(d_items));
        d_items = nullptr;
        if (k == 0) {
            CK(cudaMalloc(&d_items, sizeof(BatchItem) * items.size()));
            CK(cudaMemcpyAsync(d_items, items.data(), sizeof(BatchItem) * items.size(), cudaMemcpyHostToDevice,
                               stream));
        }
        occ = tun.ctas_per_sm;  // the persistent kernel 0: as asked
        std::vector<int> first;
        if (k == 1 || k == 2) {
            first = titem0[k];
            occ = k == 1 ? tile_occ<1>() : tile_occ<2>();
        } else if (k == 6) {
            first = xitem0[r == 4 ? 0 : 1];
            occ = r == 4 ? xtile_occ<4>() : xtile_occ<8>();
        } else {
            first = first_items(items);
        }
        for (Group& g : groups) {
            g.item0 = first[g.c0];
            g.n_items = first[g.c1] - first[g.c0];
        }
        every.n_items = first[every.c1];
        work_dirty = true;
        drop_graphs();
        CK(cudaStreamSynchronize(stream));
    }

    void drop_graphs() {
        auto drop = [](Group& g) {
            if (g.graph) cudaGraphExecDestroy(g.graph);
            g.graph = nullptr;
        };
        for (Group& g : groups) drop(g);
        drop(every);
    }

    // Brings every cavity to PC form at the shared step and refreshes the
    // cavity table (buffer parity relative to the batch clock).
    void enter() {
        for (auto* c : cv) {
            if (!c->pc_form) {
                k_collide_ref<St><<<c->grd, c->blk, 0, stream>>>(c->pop[c->cur], c->pop[c->cur ^ 1], c->rho, c->ux,
                                                                   c->uy, c->tt, c->fy, c->nut, c->G,
                                                                   c->scalars(c->time_step));
                c->check_launch();
                c->cur ^= 1;
                c->pc_form = true;
                c->ref_cached = false;
                c->time_step += 1;
                cavs_dirty = true;
            }
        }
        time_step = cv[0]->time_step;
        for (auto* c : cv)
            if (c->time_step != time_step) throw ArgError{CAV_ERR_STATE, "cavities of a batch out of step"};
        if (cavs_dirty) {
            std::vector<BatchCav<St>>& h = hcavs;
            h.resize(cv.size());
            for (size_t i = 0; i < cv.size(); ++i) {
                auto* c = cv[i];
                h[i].pop[0] = c->pop[0];
                h[i].pop[1] = c->pop[1];
                h[i].fy = c->fy;
                h[i].nut = c->nut;
                h[i].G = c->G;
                h[i].parity = (c->cur + int(time_step & 1)) & 1;
                h[i].spin_up = int(c->spin_up);
            }
            CK(cudaMemcpyAsync(d_cavs, h.data(), sizeof(BatchCav<St>) * h.size(), cudaMemcpyHostToDevice, stream));
            std::vector<TileCav<St>> t(cv.size());
            for (size_t i = 0; i < cv.size(); ++i) {
                t[i].pop[0] = h[i].pop[0];
                t[i].pop[1] = h[i].pop[1];
                t[i].fy = h[i].fy;
                t[i].nut = h[i].nut;
                t[i].acc_hot = nullptr;
                t[i].acc_cold = nullptr;
                t[i].G = h[i].G;
                t[i].parity = h[i].parity;
                t[i].spin_up = h[i].spin_up;
            }
            CK(cudaMemcpyAsync(d_tcavs, t.data(), sizeof(TileCav<St>) * t.size(), cudaMemcpyHostToDevice, stream));
            CK(cudaStreamSynchronize(stream));
            cavs_dirty = false;
            work_dirty = true;
        }
        const int k = effective_kernel(tun.kernel);
        if (work_dirty && k >= 3 && k <= 5) {
            std::vector<BatchWork<St>> w(items.size());
            for (size_t i = 0; i < items.size(); ++i) w[i] = BatchWork<St>{hcavs[items[i].cav], items[i]};
            if (d_work) CK(cudaFree(d_work));
            d_work = nullptr;
            drop_graphs();
            CK(cudaMalloc(&d_work, sizeof(BatchWork<St>) * w.size()));
            CK(cudaMemcpyAsync(d_work, w.data(), sizeof(BatchWork<St>) * w.size(), cudaMemcpyHostToDevice, stream));
            CK(cudaStreamSynchronize(stream));
            work_dirty = false;
        }
    }

    template <int V, bool WN>
    void launch_tiles(const Group& g, const long long* sdev, long long step) {
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = dim3(grid_of(g.n_items));
        cfg.blockDim = dim3(TileShape<St, V>::THREADS);
        cfg.dynamicSmemBytes = TileShape<St, V>::SMEM;
        cfg.stream = stream;
        cudaLaunchAttribute attr[1];
        attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        attr[0].val.programmaticStreamSerializationAllowed = 1;
        cfg.attrs = attr;
        cfg.numAttrs = 1;
        CK(cudaLaunchKernelEx(&cfg, k_tile<St, V, WN, false>, (const TileCav<St>*)d_tcavs,
                              (const CUtensorMap*)d_maps[V], (const TileItem*)d_titems[V] + g.item0, g.n_items,
                              (const StepScalars<A>*)d_table, int(cv.size()), step, sdev, d_err,
                              int(stall_copies)));
    }

    // The one-CTA-per-item kernels (3, 4, 5) over d_work.
    template <bool WN>
    void launch_np(const Group& g, int k, const long long* sdev, long long step) {
        const BatchWork<St>* const work = d_work + g.item0;
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = dim3(g.n_items);
        cfg.blockDim = dim3(32 * tun.rows_per_item);
        cfg.dynamicSmemBytes = 0;
        cfg.stream = stream;
        cudaLaunchAttribute attr[1];
        attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        attr[0].val.programmaticStreamSerializationAllowed = 1;
        cfg.attrs = attr;
        cfg.numAttrs = 1;
        if constexpr (has_pairs<St>::value) {
            if (k == 5) {
                CK(cudaLaunchKernelEx(&cfg, k_batch_x<St, WN>, work, (const StepScalars<float>*)d_table, table_rows,
                                      int(cv.size()), step, sdev));
                return;
            }
        }
        if constexpr (Fmt<St>::SHIFT) {
            if (k == 4) {
                cfg.blockDim = dim3(16 * tun.rows_per_item);
                CK(cudaLaunchKernelEx(&cfg, k_batch_np2<St, WN>, work, (const StepScalars<float>*)d_table, table_rows,
                                      int(cv.size()), step, sdev));
                return;
            }
        }
        CK(cudaLaunchKernelEx(&cfg, k_batch_np<St, WN>, work, (const StepScalars<A>*)d_table, table_rows,
                              int(cv.size()), step, sdev));
    }

    template <int TY, bool WN>
    void launch_xtiles(const Group& g, int slot, const long long* sdev, long long step) {
        if constexpr (is_p16<St>::value) {
            cudaLaunchConfig_t cfg = {};
            cfg.gridDim = dim3(grid_of(g.n_items));
            cfg.blockDim = dim3(TileXShape<TY>::THREADS);
            cfg.dynamicSmemBytes = TileXShape<TY>::SMEM;
            cfg.stream = stream;
            cudaLaunchAttribute attr[1];
            attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
            attr[0].val.programmaticStreamSerializationAllowed = 1;
            cfg.attrs = attr;
            cfg.numAttrs = 1;
            CK(cudaLaunchKernelEx(&cfg, k_tile_x<St, TY, WN>, (const TileCav<St>*)d_tcavs,
                                  (const CUtensorMap*)d_xmaps[slot], (const CUtensorMap*)d_fmaps[slot],
                                  (const TileItem*)d_xitems[slot] + g.item0, g.n_items, (const StepScalars<float>*)d_table,
                                  int(cv.size()), step, sdev, d_err));
        }
    }

    template <bool WN>
    void launch_kernel(const Group& g, const long long* sdev, long long step) {
        const int k = effective_kernel(tun.kernel);
        if (k == 6) {
            tun.rows_per_item == 4 ? launch_xtiles<4, WN>(g, 0, sdev, step) : launch_xtiles<8, WN>(g, 1, sdev, step);
        } else if (k >= 3) {
            launch_np<WN>(g, k, sdev, step);
        } else if (k >= 1) {
            k == 1 ? launch_tiles<1, WN>(g, sdev, step) : launch_tiles<2, WN>(g, sdev, step);
        } else {
            k_batch<St, WN><<<grid_of(g.n_items), BATCH_THREADS, 0, stream>>>(
                d_cavs, d_items + g.item0, g.n_items, d_table, int(cv.size()), step, sdev);
        }
    }

    void launch(const Group& g, bool write_nut, const long long* sdev, long long step) {
        write_nut ? launch_kernel<true>(g, sdev, step) : launch_kernel<false>(g, sdev, step);
        ++launches;
        CK(cudaGetLastError());
    }

    cudaGraphExec_t get_graph(Group& g) {
        if (g.graph) return g.graph;
        const int64_t l0 = launches;
        CK(cudaStreamBeginCapture(stream, cudaStreamCaptureModeThreadLocal));
        for (int j = 0; j < GRAPH_STEPS; ++j) launch(g, false, step_dev, j);
        k_add_step<<<1, 1, 0, stream>>>(step_dev, GRAPH_STEPS);
        cudaGraph_t gr;
        CK(cudaStreamEndCapture(stream, &gr));
        launches = l0;
        CK(cudaGraphInstantiate(&g.graph, gr, 0));
        cudaGraphDestroy(gr);
        return g.graph;
    }

    void advance_cavities(int64_t k) {
        for (auto* c : cv) {
            if (k & 1) c->cur ^= 1;
            c->time_step += k;
            c->ref_cached = false;
        }
        time_step += k;
    }

    void step(int64_t n) override {
        if (n <= 0) return;
        bool entered_with_collide = false;
        for (auto* c : cv) entered_with_collide |= !c->pc_form;
        enter();  // may run one collision (the first step from a REF state)
        if (entered_with_collide) n -= 1;
        if (n <= 0) return;
        if (groups.size() > 1 && n > ungrouped_steps()) {
            for (Group& g : groups) step_group(g, n);
        } else {
            step_group(every, n);
        }
        advance_cavities(n);
    }

    // The longest call that is run as one launch per step over all cavities.  A
    // group pays a launch's start and last wave at every step and gains from its
    // second step on, and only where the kernel waits for memory: the TMA-staged
    // kernels (1, 6; 2 in 16 bits) and the one-node kernel 3 in 16 bits, which is
    // bound by issue, do not.  B200, us per step of an n-step call, one launch /
    // groups (64-cavity sweep; 160 cavities):
    //   FP32 kernel 3    n 1: 80.0 / 93.2   2: 71.3 / 75.0   3: 66.5 / 62.9   (160) 2: 169 / 179   3: 164 / 158
    //   f16sr kernel 5   n 1: 71.4 / 69.2   2: 54.1 / 56.5   3: 52.2 / 51.9   (160) 2: 127 / 137   3: 125 / 127
    //   f16sr kernel 4   n 3: 56.4 / 56.3   6: 52.7 / 51.9   64: 49.5 / 47.6  (160) 4: 132 / 139   16: 128 / 130
    //   f16sr kernel 3   n 1: 76.9 / 80.6   8: 53.6 / 55.5   64: 51.2 / 52.2  (160) 64: 135 / 139
    //   f16sr kernel 6   n 1: 65.8 / 73.8   8: 44.1 / 49.7   64: 42.1 / 45.8  (160) 64: 113 / 122
    //   FP32 kernel 0    n 8: 78.9 / 80.5   16: 77.8 / 77.0  64: 77.1 / 74.5  (160) 16: 194 / 195
    //   FP32 kernel 2    n 4: 101 / 102     8: 99.6 / 93.0   64: 98.5 / 85.6  (160) 6: 243 / 242
    int64_t ungrouped_steps() const {
        constexpr bool p16 = is_p16<St>::value;
        constexpr int64_t any = std::numeric_limits<int64_t>::max();
        switch (effective_kernel(tun.kernel)) {
            case 0: return 16;
            case 2: return p16 ? any : 6;
            case 3: return p16 ? any : 2;
            case 4: return p16 ? 4 : 2;
            case 5: return 2;
            default: return any;
        }
    }

    // n steps of one group from the shared step (its cavities in PC form).
    void step_group(Group& g, int64_t n) {
        int64_t s = time_step;
        if (n > GRAPH_STEPS && step_dev_val != s) {
            k_set_step<<<1, 1, 0, stream>>>(step_dev, s);
            CK(cudaGetLastError());
            ++launches;
            step_dev_val = s;
        }
        while (n > 0) {
            if (n > GRAPH_STEPS) {
                CK(cudaGraphLaunch(get_graph(g), stream));
                launches += GRAPH_STEPS + 1;
                step_dev_val += GRAPH_STEPS;
                s += GRAPH_STEPS;
                n -= GRAPH_STEPS;
            } else {
                launch(g, n == 1, nullptr, s);
                s += 1;
                n -= 1;
            }
        }
    }

    double time_steps(int steps) override {
        enter();
        cudaEvent_t a, b;
        CK(cudaEventCreate(&a));
        CK(cudaEventCreate(&b));
        // warm-up; the graphs only where the timed steps replay them
        step(steps > GRAPH_STEPS ? GRAPH_STEPS + 1 : 4);
        CK(cudaEventRecord(a, stream));
        step(steps);
        CK(cudaEventRecord(b, stream));
        CK(cudaEventSynchronize(b));
        check_err();
        float ms = 0.f;
        CK(cudaEventElapsedTime(&ms, a, b));
        cudaEventDestroy(a);
        cudaEventDestroy(b);
        return ms;
    }

    // A tile CTA that gave up waiting for its copies (k_tile) sets *d_err;
    // reported once, then cleared (the steps of that launch are lost).
    void check_err() {
        CK(cudaMemcpyAsync(h_err, d_err, sizeof(unsigned), cudaMemcpyDeviceToHost, stream));
        CK(cudaStreamSynchronize(stream));
        if (*h_err) {
            *h_err = 0;
            CK(cudaMemsetAsync(d_err, 0, sizeof(unsigned), stream));
            CK(cudaStreamSynchronize(stream));
            throw ArgError{CAV_ERR_TIMEOUT, "a tile copy did not complete within its bounded wait"};
        }
    }

    void set_stall_copies(bool on) override {
        CK(cudaStreamSynchronize(stream));
        stall_copies = on;
        drop_graphs();
    }

    void sync() override { check_err(); }
};

}  // namespace cav
