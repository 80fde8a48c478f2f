// kwg_uneven.cu -- kwg_fd1d_price_uneven: a batch in which every option has its own
// x-grid size and number of time levels.
//
// The reference prices one grid shape per Fd1d_Pricer::init (src/Pricer/kwFd1d.cpp:
// 15-16), so a mixed portfolio needs one call per shape.  Here the whole batch is
// one pass over the device:
//   * dedup by (t, r, q, z, e, w, x_dim, t_dim), like src/Pricer/kwFd1d.cpp:28-65
//     with the grid added to the key;
//   * FP64 (thread per option): PDEs of equal x_dim are packed 32 to a tile, sorted
//     by t_dim so that the lanes of a tile finish together, and all tiles run in ONE
//     persistent launch whose queue hands out the longest tiles first; each lane
//     steps its own t_dim - 1 times.  The device sequence (H2D copy, kernels, D2H copy) is
//     captured once into a CUDA graph and replayed while the batch layout stays the same;
//   * warp-per-PDE solvers (FP32, FP64 in pair arithmetic, or KWG_SOLVER_PCR): the options
//     are split into one bucket per nodes-per-lane count, and every bucket is prepared, solved and
//     copied on a stream of its own, the heaviest first (price_buckets).
#include <algorithm>
#include <chrono>
#include <cmath>
#include <cstdint>
#include <cstdio>
#include <cstring>
#include <new>
#include <numeric>
#include <vector>

#include <cuda_runtime.h>

#include "fd1d_kernels.h"
#include "fp64_route.h"
#include "host_dedup.h"
#include "kwg.h"
#include "kwg_ctx.h"

using namespace kwgi;

namespace {

struct UnevenLayout {
    size_t t, z, r, q, px, pt, w, e, s, k, pde, tiles, rows, in_bytes;
    size_t prices, status, out_bytes, pde_status, total;
};

UnevenLayout uneven_layout(size_t m, size_t n, size_t ntiles)
{
    UnevenLayout L;
    size_t o = 0;
    auto take = [&](size_t bytes) {
        const size_t at = o;
        o = align_up(o + bytes, 256);
        return at;
    };
    L.t = take(m * 8);
    L.z = take(m * 8);
    L.r = take(m * 8);
    L.q = take(m * 8);
    L.px = take(m * 4);
    L.pt = take(m * 4);
    L.w = take(m);
    L.e = take(m);
    L.s = take(n * 8);
    L.k = take(n * 8);
    L.pde = take(n * 4);
    L.tiles = take(ntiles * sizeof(kwg::TileDesc));
    L.rows = take(m * sizeof(long long));
    L.in_bytes = o;
    L.prices = take(n * 8);
    L.status = take(n * 4);
    L.out_bytes = o - L.prices;
    L.pde_status = take(m * 4);
    L.total = o;
    return L;
}

constexpr int kBuckets = sizeof(kwg_ctx::buckets) / sizeof(kwg_ctx::Bucket);

// Warp-per-PDE solvers.  Preparing a batch (dedup, sort by work, packing) takes the host ~85 ns per
// option: 11 of the 52 ms of 131072 options in FP32 when the whole batch was prepared before
// the first kernel, and the solves of the buckets waited for one another's last PDEs.  By buckets, all but the
// first one's preparation hides behind the device, and a bucket's tail behind the
// next one's start: 42.8 ms (FP64: 143.9 -> 129.9).  With profiling on all run on the context's stream, one after
// the other.
int price_buckets(kwg_ctx* ctx, const kwg_option* opts, const int32_t* x_dims, const int32_t* t_dims, size_t n,
                  const kwg_fd1d_params& q, const kwg_ctx::Tuned& tn, bool pair, const kwg::Fp64Batch* costs,
                  double* prices, int32_t* status)
{
    auto mlane = [&](int x) {
        return q.precision == KWG_FP32 || pair ? kwg::fd1d_fp32_nodes_per_lane(x) : kwg::fd1d_pcr64_nodes_per_lane(x);
    };
    // options by bucket, in the caller's order within one
    struct Part {
        size_t begin = 0, end = 0, at = 0;
        uint64_t work = 0, nodes = 0;
        UnevenLayout L;
    } part[kBuckets];
    std::vector<uint8_t> id(n);
    for (size_t i = 0; i < n; ++i) {
        const int M = mlane(x_dims[i]);
        int b = 0;
        while (b < kBuckets - 1 && (2 << b) < M) ++b;
        if (M < 0) return set_err(ctx, KWG_ERR_INVALID, "kwg: grid too large for the chosen solver");
        id[i] = (uint8_t)b;
        ++part[b].end;
        part[b].work += (uint64_t)x_dims[i] * (uint64_t)(t_dims[i] - 1);
        part[b].nodes += (uint64_t)x_dims[i];
    }
    size_t off = 0;
    for (Part& p : part) {
        p.begin = p.at = off;
        off = p.end += off;
    }
    std::vector<uint32_t> order(n);
    for (size_t i = 0; i < n; ++i) order[part[id[i]].at++] = (uint32_t)i;
    // The heaviest bucket first.  The others by work as well, but in pair arithmetic upwards: a
    // bucket's rescue launch (fd1d_pair64.cu), one PDE's FP64 latency however short its list, then runs
    // beside the next bucket (in FP32, which has none, 1.86 -> 1.97 ms for 4000 options).  In large batches the
    // heavy buckets' own tails weigh as much: downwards / upwards 8000 options 15.2 / 12.3 ms, 16000 22.8 / 18.9, 32000
    // 34.0 / 33.5, 48000 49.7 / 51.7, 131072 132.9 / 132.9.
    int by_work[kBuckets];
    std::iota(by_work, by_work + kBuckets, 0);
    std::stable_sort(by_work, by_work + kBuckets, [&](int a, int b) { return part[a].work > part[b].work; });
    if (pair && n < 32768) std::reverse(by_work + 1, by_work + kBuckets);

    // Buffers of the later buckets before the first launch, as growing one later would wait for the solves in
    // flight: at the size they have with the first bucket's share of distinct PDEs and a tenth.  Batches
    // beyond 2 GB of rows, what does not fit, and buckets with a larger share grow one by one.
    auto reserve = [&](int first, double distinct) {
        size_t m[kBuckets], nodes[kBuckets], rows = 0;
        for (int b = 0; b < kBuckets; ++b) {
            const size_t nb = part[b].end - part[b].begin;
            m[b] = std::min(nb, (size_t)(1.1 * distinct * (double)nb) + 32);
            nodes[b] = std::min((size_t)part[b].nodes, (size_t)(1.1 * distinct * (double)part[b].nodes) + 32 * ((size_t)64 << b));
            rows += nodes[b] * sizeof(double);
        }
        for (int b = 0; b < kBuckets && rows <= 2000000000ull; ++b) {
            const size_t nb = part[b].end - part[b].begin;
            kwg_ctx::Bucket& bk = ctx->buckets[b];
            if (nb == 0 || b == first) continue;
            const size_t io = uneven_layout(m[b], nb, 0).total,
                         work = pair ? kwg::fd1d_pair64_work_bytes((int)m[b], (long long)nodes[b]) : nodes[b] * sizeof(double);
            if (ensure_host(ctx, &bk.h_io, &bk.h_io_bytes, io) ||
                ensure_device(ctx, &bk.d_io, &bk.io_bytes, align_up(io, 256) + 4 * sizeof(int)) ||
                ensure_device(ctx, &bk.d_work, &bk.work_bytes, work)) {
                ctx->err.clear();
                cudaGetLastError();
                break;
            }
        }
    };

    std::vector<int32_t> asset2pde, pde_slot;
    std::vector<uint32_t> pde2asset;
    std::vector<std::pair<uint64_t, uint32_t>> kv;
    auto prepare = [&](int bi) -> int {
        const Part& p = part[bi];
        kwg_ctx::Bucket& bk = ctx->buckets[bi];
        const uint32_t* const idx = order.data() + p.begin;
        const size_t nb = p.end - p.begin;
        const size_t m = kwg::dedup_host(opts, nb, x_dims, t_dims, asset2pde, pde2asset, idx);
        if (bi == by_work[0]) reserve(bi, (double)m / (double)nb);
        // node-steps descending (x_dim <= 2048 here, so node-steps < 2^43), ties by PDE number
        kv.resize(m);
        int x_max = 0, x_min = INT32_MAX;
        long long nodes = 0;
        for (size_t i = 0; i < m; ++i) {
            const int x = x_dims[pde2asset[i]];
            kv[i] = {((1ull << 50) - 1) - (uint64_t)x * (uint64_t)(t_dims[pde2asset[i]] - 1), (uint32_t)i};
            x_max = std::max(x_max, x);
            x_min = std::min(x_min, x);
            nodes += x;
        }
        kwg::radix_sort_pairs(kv);
        UnevenLayout& L = part[bi].L;
        L = uneven_layout(m, nb, 0);
        const size_t counters = align_up(L.total, 256), wbytes = pair ? kwg::fd1d_pair64_work_bytes((int)m, nodes)
                                                                      : (size_t)nodes * sizeof(double);
        if (int rc = ensure_host(ctx, &bk.h_io, &bk.h_io_bytes, L.total)) return rc;
        if (int rc = ensure_device(ctx, &bk.d_io, &bk.io_bytes, counters + 4 * sizeof(int))) return rc;
        if (int rc = ensure_device(ctx, &bk.d_work, &bk.work_bytes, wbytes)) return rc;
        if (!bk.stream) KWG_CUDA(ctx, cudaStreamCreateWithFlags(&bk.stream, cudaStreamNonBlocking));
        char *h = (char*)bk.h_io, *io = (char*)bk.d_io;
        pde_slot.resize(m);
        long long row = 0;
        for (size_t sl = 0; sl < m; ++sl) {
            const uint32_t at = pde2asset[kv[sl].second];
            const kwg_option& o = opts[at];
            pde_slot[kv[sl].second] = (int32_t)sl;
            ((double*)(h + L.t))[sl] = o.t;
            ((double*)(h + L.z))[sl] = o.z;
            ((double*)(h + L.r))[sl] = o.r;
            ((double*)(h + L.q))[sl] = o.q;
            ((int32_t*)(h + L.px))[sl] = x_dims[at];
            ((int32_t*)(h + L.pt))[sl] = t_dims[at];
            ((int8_t*)(h + L.w))[sl] = o.w;
            ((uint8_t*)(h + L.e))[sl] = o.e;
            ((long long*)(h + L.rows))[sl] = row;
            row += x_dims[at];
        }
        for (size_t i = 0; i < nb; ++i) {
            ((double*)(h + L.s))[i] = opts[idx[i]].s;
            ((double*)(h + L.k))[i] = opts[idx[i]].k;
            ((int32_t*)(h + L.pde))[i] = pde_slot[asset2pde[i]];
        }
        kwg::PdeBatch b;
        b.t = (const double*)(io + L.t);
        b.z = (const double*)(io + L.z);
        b.r = (const double*)(io + L.r);
        b.q = (const double*)(io + L.q);
        b.w = (const int8_t*)(io + L.w);
        b.e = (const uint8_t*)(io + L.e);
        b.m = b.m_pad = (int)m;
        kwg::AssetBatch a;
        a.s = (const double*)(io + L.s);
        a.k = (const double*)(io + L.k);
        a.pde = (const int32_t*)(io + L.pde);
        a.n = (int)nb;
        kwg::Fd1dShape sh = make_shape(&q);
        sh.x_dim = x_max;
        sh.block_warps = tn.block_warps;
        sh.option_warps = tn.option_warps;
        sh.sm_blocks = tn.sm_blocks;
        sh.pde_x = (const int32_t*)(io + L.px);
        sh.pde_t = (const int32_t*)(io + L.pt);
        sh.row_off = (const long long*)(io + L.rows);
        sh.full_lanes = x_min == kwg::kTile * mlane(x_max);  // all fill the lanes
        double *v = (double*)bk.d_work, *d_prices = (double*)(io + L.prices);
        int32_t *d_status = (int32_t*)(io + L.status), *d_pde_status = (int32_t*)(io + L.pde_status);
        int* const d_counters = (int*)(io + counters);
        const cudaStream_t st = ctx->profiling ? ctx->stream : bk.stream;
        KWG_CUDA(ctx, cudaMemcpyAsync(io, h, L.in_bytes, cudaMemcpyHostToDevice, st));
        const kwg::SolveEvents* ev = ctx->next_events();
        const bool fp64_steps = pair && costs[bi].fp64_beside_others();
        const int r =
            fp64_steps ? kwg::fd1d_pcr64_half_launch(b, a, sh, v, d_pde_status, d_counters, d_prices, d_status,
                                                     ctx->device, st, ev)
            : pair ? kwg::fd1d_pair64_launch(b, a, sh, v, (int32_t*)(v + nodes), d_pde_status, d_counters, d_prices,
                                           d_status, ctx->device, st, ev)
            : q.precision == KWG_FP32 ? kwg::fd1d_fp32_launch(b, a, sh, v, d_pde_status, d_counters, d_prices,
                                                              d_status, ctx->device, st, ev)
                                      : kwg::fd1d_pcr64_launch(b, a, sh, v, d_pde_status, d_counters, d_prices,
                                                               d_status, ctx->device, st, ev);
        if (r < 0) return set_err(ctx, KWG_ERR_INVALID, "kwg: grid too large for the chosen solver");
        ctx->launches += r;
        KWG_CUDA(ctx, cudaGetLastError());
        KWG_CUDA(ctx, cudaMemcpyAsync(h + L.prices, io + L.prices, L.out_bytes, cudaMemcpyDeviceToHost, st));
        return KWG_OK;
    };

    int rc = KWG_OK;
    for (int bi : by_work) {
        if (rc == KWG_OK && part[bi].end > part[bi].begin) {
            try {
                rc = prepare(bi);
            } catch (const std::bad_alloc&) {  // buckets in flight are drained below
                rc = set_err(ctx, KWG_ERR_INVALID, "kwg: out of host memory");
            }
        }
    }
    // results, bucket by bucket while later ones run; after an error the streams are drained
    for (int bi : by_work) {
        const Part& p = part[bi];
        kwg_ctx::Bucket& bk = ctx->buckets[bi];
        if (p.end == p.begin || !bk.stream) continue;
        const cudaError_t e = cudaStreamSynchronize(ctx->profiling ? ctx->stream : bk.stream);
        if (rc != KWG_OK) continue;
        if (e != cudaSuccess) {
            rc = cuda_err(ctx, e, "kwg: uneven batch");
            continue;
        }
        const double* hp = (const double*)((char*)bk.h_io + p.L.prices);
        const int32_t* hs = (const int32_t*)((char*)bk.h_io + p.L.status);
        for (size_t i = p.begin; i < p.end; ++i) {
            prices[order[i]] = hp[i - p.begin];
            status[order[i]] = hs[i - p.begin];
        }
    }
    return rc;
}

// Strict mode: the first asset without a price is an error.
int check_strict(kwg_ctx* ctx, const int32_t* status, size_t n)
{
    for (size_t i = 0; i < n; ++i) {
        if (status[i] == KWG_STATUS_OK) continue;
        char msg[256];
        std::snprintf(msg, sizeof msg, "Fd1dGpu_Pricer::price: asset %zu: %s", i,
                      status[i] == KWG_STATUS_OUT_OF_GRID ? "not in grid range" : "failed");
        return set_err(ctx, status[i] == KWG_STATUS_OUT_OF_GRID ? KWG_ERR_OUT_OF_GRID : KWG_ERR_SOLVER, msg);
    }
    return KWG_OK;
}

uint64_t mix(uint64_t h, uint64_t v)
{
    h ^= v + 0x9e3779b97f4a7c15ull + (h << 6) + (h >> 2);
    return h;
}

}  // namespace

extern "C" int kwg_fd1d_price_uneven(kwg_ctx* ctx, const kwg_option* opts, const int32_t* x_dims,
                                     const int32_t* t_dims, size_t n, const kwg_fd1d_params* p, double* prices,
                                     int32_t* status)
{
    if (!ctx) return KWG_ERR_INVALID;
    ctx->err.clear();
    ctx->launches = 0;
    if (!p) return set_err(ctx, KWG_ERR_INVALID, "kwg: null params");
    if (n == 0) return KWG_OK;
    if (!opts || !x_dims || !t_dims || !prices)
        return set_err(ctx, KWG_ERR_INVALID, "kwg: null options, grid sizes or prices");
    if (n > (size_t)INT32_MAX / 4) return set_err(ctx, KWG_ERR_INVALID, "kwg: batch too large");
    int x_max = 0, t_max = 0;
    for (size_t i = 0; i < n; ++i) {
        if (x_dims[i] < 3 || t_dims[i] < 2) {
            char msg[160];
            std::snprintf(msg, sizeof msg, "kwg: option %zu: x_dim must be >= 3 and t_dim >= 2 (got %d, %d)", i,
                          x_dims[i], t_dims[i]);
            return set_err(ctx, KWG_ERR_INVALID, msg);
        }
        x_max = std::max(x_max, (int)x_dims[i]);
        t_max = std::max(t_max, (int)t_dims[i]);
    }
    kwg_fd1d_params q = *p;
    q.x_dim = x_max;
    q.t_dim = t_max;
    if (int rc = check_params(ctx, &q)) return rc;
    // launch choices: the explicit ones, else what kwg_autotune_uneven recorded for
    // uneven batches of this precision and size, else the on-chip solvers with warps by the
    // bucket's size, or (theta != 1/2, more than 2048 nodes, and where the cost model of fp64_route.h
    // says so) Thomas.  PDEs left over by pair arithmetic bring the model in where that is recorded too.
    kwg_ctx::Tuned tn;
    kwg::Fp64Batch costs[kBuckets];
    for (kwg::Fp64Batch& c : costs) c.uniform = std::isinf(q.density);
    {
        const auto it = ctx->tuned.find(tune_key(&q, 0, 0, (long long)n));
        const bool recorded = it != ctx->tuned.end();
        if (recorded) tn = it->second;
        const bool may_pair = pair64_ok(&q) && q.solver != KWG_SOLVER_THOMAS &&
                              !(q.solver == KWG_SOLVER_AUTO && recorded && tn.solver == KWG_SOLVER_THOMAS);
        if (may_pair)  // every option a PDE of its own
            for (size_t i = 0; i < n; ++i)
                costs[kwg::Fp64Batch::size_of(x_dims[i])].add(
                    1, x_dims[i], t_dims[i] - 1,
                    kwg::pair64_leaves(opts[i].t, opts[i].z, opts[i].r, opts[i].q, opts[i].w, q.scale));
        if (may_pair && q.solver == KWG_SOLVER_AUTO) {
            kwg::Fp64Batch b(std::isinf(q.density));
            for (const kwg::Fp64Batch& c : costs) b.add(c);
            tn.solver = KWG_SOLVER_PCR;
            if ((!recorded || b.any_left()) && b.best() == kwg::Fp64Route::kStream) {
                tn.solver = KWG_SOLVER_THOMAS;
                if (b.few_long_chains()) {
                    tn.block_warps = 4;
                    tn.sm_blocks = 1;
                }
            }
        }
        if (q.precision == KWG_FP64 && q.solver == KWG_SOLVER_AUTO &&
            (tn.solver != KWG_SOLVER_PCR || pair64_ok(&q) || kwg::fd1d_pcr64_nodes_per_lane(x_max) > 0))
            q.solver = tn.solver;
        if (q.block_warps || q.sm_blocks) {
            if (q.block_warps) tn.block_warps = q.block_warps;
            tn.sm_blocks = q.sm_blocks;
        }
        if (q.option_warps) tn.option_warps = q.option_warps;
    }
    const bool pcr = q.precision == KWG_FP32 || q.solver == KWG_SOLVER_PCR;
    const bool pair = q.solver == KWG_SOLVER_PCR && pair64_ok(&q);
    KWG_CUDA(ctx, cudaSetDevice(ctx->device));
    auto on_chip = [&](bool in_pairs) {
        std::vector<int32_t> own;
        if (!status) {
            own.resize(n);
            status = own.data();
        }
        const int rc = price_buckets(ctx, opts, x_dims, t_dims, n, q, tn, in_pairs, costs, prices, status);
        return rc == KWG_OK && p->strict ? check_strict(ctx, status, n) : rc;
    };
    if (pcr) return on_chip(pair);

    // 1. dedup by (t, r, q, z, e, w, x_dim, t_dim)
    std::vector<int32_t> asset2pde;
    std::vector<uint32_t> pde2asset;
    const size_t m = kwg::dedup_host(opts, n, x_dims, t_dims, asset2pde, pde2asset);
    auto xd = [&](size_t pde) { return x_dims[pde2asset[pde]]; };
    auto td = [&](size_t pde) { return t_dims[pde2asset[pde]]; };

    // 2. layout: slot order and tiles
    std::vector<uint32_t> slot_pde;          // slot -> PDE (replicas pad tiles)
    std::vector<int32_t> pde_slot(m, -1);    // PDE -> its first slot
    std::vector<kwg::TileDesc> tiles;
    long long node_lanes = 0;
    // PDEs in layout order: sorted on one packed integer key per PDE (ties by PDE
    // number, so the layout is deterministic)
    std::vector<uint32_t> by(m);
    auto sort_by = [&](auto packed_key) {
        std::vector<std::pair<uint64_t, uint32_t>> kv(m);
        for (size_t i = 0; i < m; ++i) kv[i] = {packed_key((uint32_t)i), (uint32_t)i};
        kwg::radix_sort_pairs(kv);
        for (size_t i = 0; i < m; ++i) by[i] = kv[i].second;
    };
    // x_dim ascending, t_dim descending
    sort_by([&](uint32_t p) { return (uint64_t)(uint32_t)xd(p) << 32 | (uint32_t)(INT32_MAX - td(p)); });
    struct Chunk {
        size_t begin, count;
        int x, tmax;
    };
    std::vector<Chunk> chunks;
    for (size_t i = 0; i < m;) {
        size_t j = i;
        while (j < m && xd(by[j]) == xd(by[i])) ++j;
        for (size_t c = i; c < j; c += kwg::kTile) {
            const size_t cnt = std::min((size_t)kwg::kTile, j - c);
            chunks.push_back({c, cnt, xd(by[c]), td(by[c])});  // sorted: first has the largest t_dim
        }
        i = j;
    }
    std::stable_sort(chunks.begin(), chunks.end(), [](const Chunk& a, const Chunk& b) {
        return (long long)a.x * (a.tmax - 1) > (long long)b.x * (b.tmax - 1);
    });
    for (const Chunk& c : chunks) {
        tiles.push_back(kwg::TileDesc{c.x, c.tmax, node_lanes});
        node_lanes += (long long)kwg::kTile * c.x;
        for (int l = 0; l < kwg::kTile; ++l) {
            const uint32_t pde = by[c.begin + std::min((size_t)l, c.count - 1)];
            if (pde_slot[pde] < 0) pde_slot[pde] = (int32_t)slot_pde.size();
            slot_pde.push_back(pde);
        }
    }
    const size_t ms = slot_pde.size();

    // 3. pack inputs into pinned memory
    const UnevenLayout L = uneven_layout(ms, n, tiles.size());
    const size_t wbytes = kwg::fd1d_fp64_work_bytes_nl((int)ms, node_lanes);
    if (p->solver == KWG_SOLVER_AUTO && pair64_ok(&q) && ensure_device(ctx, &ctx->d_work, &ctx->work_bytes, wbytes)) {
        // no room for the streaming solver's 72 bytes per node: on chip it is a ninth
        ctx->err.clear();
        cudaGetLastError();
        return on_chip(true);
    }
    if (int rc = ensure_host(ctx, &ctx->h_io, &ctx->h_io_bytes, L.total)) return rc;
    // the graph bakes in device addresses: grow buffers before deciding on replay
    if (int rc = ensure_device(ctx, &ctx->d_io, &ctx->io_bytes, L.total)) return rc;
    if (int rc = ensure_device(ctx, &ctx->d_work, &ctx->work_bytes, wbytes)) return rc;
    char* h = (char*)ctx->h_io;
    for (size_t sl = 0; sl < ms; ++sl) {
        const kwg_option& o = opts[pde2asset[slot_pde[sl]]];
        ((double*)(h + L.t))[sl] = o.t;
        ((double*)(h + L.z))[sl] = o.z;
        ((double*)(h + L.r))[sl] = o.r;
        ((double*)(h + L.q))[sl] = o.q;
        ((int32_t*)(h + L.px))[sl] = xd(slot_pde[sl]);
        ((int32_t*)(h + L.pt))[sl] = td(slot_pde[sl]);
        ((int8_t*)(h + L.w))[sl] = o.w;
        ((uint8_t*)(h + L.e))[sl] = o.e;
    }
    for (size_t i = 0; i < n; ++i) {
        ((double*)(h + L.s))[i] = opts[i].s;
        ((double*)(h + L.k))[i] = opts[i].k;
        ((int32_t*)(h + L.pde))[i] = pde_slot[asset2pde[i]];
    }
    if (!tiles.empty()) std::memcpy(h + L.tiles, tiles.data(), tiles.size() * sizeof(kwg::TileDesc));

    // 4. the device sequence, as a CUDA graph when not profiling
    char* io = (char*)ctx->d_io;
    kwg::PdeBatch b;
    b.t = (const double*)(io + L.t);
    b.z = (const double*)(io + L.z);
    b.r = (const double*)(io + L.r);
    b.q = (const double*)(io + L.q);
    b.w = (const int8_t*)(io + L.w);
    b.e = (const uint8_t*)(io + L.e);
    b.m = (int)ms;
    b.m_pad = (int)ms;
    kwg::AssetBatch a;
    a.s = (const double*)(io + L.s);
    a.k = (const double*)(io + L.k);
    a.pde = (const int32_t*)(io + L.pde);
    a.n = (int)n;
    kwg::Fd1dShape sh = make_shape(&q);
    sh.block_warps = tn.block_warps;
    sh.sm_blocks = tn.sm_blocks;
    sh.pde_x = (const int32_t*)(io + L.px);
    sh.pde_t = (const int32_t*)(io + L.pt);
    sh.tiles = (const kwg::TileDesc*)(io + L.tiles);
    sh.node_lanes = node_lanes;
    double* d_prices = (double*)(io + L.prices);
    int32_t* d_status = (int32_t*)(io + L.status);
    int32_t* d_pde_status = (int32_t*)(io + L.pde_status);

    auto enqueue = [&](cudaStream_t st) -> int {
        cudaMemcpyAsync(ctx->d_io, ctx->h_io, L.in_bytes, cudaMemcpyHostToDevice, st);
        const int blocks =
            kwg::fd1d_fp64_solve_blocks((int)tiles.size(), ctx->device, sh.block_warps, sh.sm_blocks);
        const int launches = kwg::fd1d_fp64_launch(b, a, sh, (double*)ctx->d_work, d_pde_status, ctx->d_counter, d_prices,
                                                   d_status, blocks, st, ctx->next_events());
        cudaMemcpyAsync(h + L.prices, io + L.prices, L.out_bytes, cudaMemcpyDeviceToHost, st);
        return launches;
    };

    uint64_t sig = 0x5eed;
    for (uint64_t v : {(uint64_t)q.precision, (uint64_t)sh.block_warps, (uint64_t)sh.sm_blocks, (uint64_t)n, (uint64_t)ms,
                       (uint64_t)tiles.size(), (uint64_t)node_lanes, (uint64_t)(uintptr_t)ctx->d_io,
                       (uint64_t)(uintptr_t)ctx->d_work, (uint64_t)(uintptr_t)ctx->h_io})
        sig = mix(sig, v);
    for (double v : {q.theta, q.scale, q.density}) {
        uint64_t u;
        std::memcpy(&u, &v, 8);
        sig = mix(sig, u);
    }
    if (ctx->profiling) {
        const int r = enqueue(ctx->stream);
        if (r < 0) return set_err(ctx, KWG_ERR_INVALID, "kwg: grid too large for the chosen solver");
        ctx->launches += r;
        KWG_CUDA(ctx, cudaGetLastError());
    } else {
        if (!ctx->graph_exec || ctx->graph_sig != sig) {
            if (ctx->graph_exec) {
                cudaGraphExecDestroy(ctx->graph_exec);
                ctx->graph_exec = nullptr;
            }
            cudaGraph_t graph = nullptr;
            KWG_CUDA(ctx, cudaStreamBeginCapture(ctx->stream, cudaStreamCaptureModeThreadLocal));
            const int r = enqueue(ctx->stream);
            const cudaError_t ce = cudaStreamEndCapture(ctx->stream, &graph);
            if (r < 0) {
                if (graph) cudaGraphDestroy(graph);
                return set_err(ctx, KWG_ERR_INVALID, "kwg: grid too large for the chosen solver");
            }
            if (ce != cudaSuccess) return cuda_err(ctx, ce, "cudaStreamEndCapture");
            const cudaError_t ie = cudaGraphInstantiate(&ctx->graph_exec, graph, 0);
            cudaGraphDestroy(graph);
            if (ie != cudaSuccess) return cuda_err(ctx, ie, "cudaGraphInstantiate");
            ctx->graph_sig = sig;
            ctx->graph_launches = r;
        }
        KWG_CUDA(ctx, cudaGraphLaunch(ctx->graph_exec, ctx->stream));
        ctx->launches += ctx->graph_launches;
    }
    KWG_CUDA(ctx, cudaStreamSynchronize(ctx->stream));

    // 5. results and strict mode
    const double* hp = (const double*)(h + L.prices);
    const int32_t* hs = (const int32_t*)(h + L.status);
    std::memcpy(prices, hp, n * sizeof(double));
    if (status) std::memcpy(status, hs, n * sizeof(int32_t));
    return p->strict ? check_strict(ctx, hs, n) : KWG_OK;
}

extern "C" int kwg_autotune_uneven(kwg_ctx* ctx, const kwg_option* opts, const int32_t* x_dims,
                                   const int32_t* t_dims, size_t n, const kwg_fd1d_params* p, kwg_tuning* out)
{
    if (!ctx) return KWG_ERR_INVALID;
    ctx->err.clear();
    if (!p || !opts || !x_dims || !t_dims || n == 0 || n > (size_t)INT32_MAX / 4)
        return set_err(ctx, KWG_ERR_INVALID, "kwg_autotune_uneven: bad arguments");
    int x_max = 0;
    for (size_t i = 0; i < n; ++i) x_max = std::max(x_max, (int)x_dims[i]);
    std::vector<double> prices(n);
    const bool pcr_ok = kwg::fd1d_pcr64_nodes_per_lane(x_max) > 0;
    const uint64_t key = tune_key(p, 0, 0, (long long)n);
    ctx->tuned[key] = kwg_ctx::Tuned();
    ctx->tuned[key].solver = KWG_SOLVER_PCR;
    kwg_fd1d_params widest = *p;
    widest.x_dim = x_max;
    auto call = [&](const kwg_fd1d_params& q) {
        return kwg_fd1d_price_uneven(ctx, opts, x_dims, t_dims, n, &q, prices.data(), nullptr);
    };
    kwg_ctx::Tuned best = tune(ctx, p, 0, pcr_ok, pair64_ok(&widest), call, out);
    if (p->precision == KWG_FP32) {
        // One number of warps for all buckets against each bucket's own by its size.  Whole calls
        // decide: the candidates' solves were timed one after the other, and buckets that run side
        // by side want fewer warps (5321 options: 8 warps 3.0 ms a call, by size 2.8).
        kwg_fd1d_params q = *p;
        q.strict = 0;
        auto wall = [&](int warps) {
            q.option_warps = warps;
            double ms = -1.;
            for (int i = 0; i < 4; ++i) {
                const auto t0 = std::chrono::steady_clock::now();
                if (call(q) != KWG_OK) return -1.;
                const double d = std::chrono::duration<double, std::milli>(std::chrono::steady_clock::now() - t0).count();
                if (ms < 0. || d < ms) ms = d;
            }
            return ms;
        };
        const double fixed = wall(best.option_warps), own = wall(0);
        if (own >= 0. && own <= 1.02 * fixed) {
            best.option_warps = 0;
            if (out) out->option_warps = 0;
        }
    }
    ctx->tuned[key] = best;
    ctx->err.clear();
    return KWG_OK;
}
