// fp64_route.h -- which FP64 solver takes a batch at theta = 1/2 on up to 2048 nodes: a cost
// model of the three, shared by every entry point.
//   kPair    pair arithmetic on chip; PDEs that it leaves over (fd1d_pair64.cu) go through its setup and
//            then to the warp-per-PDE FP64 kernel, in a launch of their own;
//   kOnChip  the warp-per-PDE FP64 kernel for all of them;
//   kStream  the streaming solver, one thread per PDE.
// Without PDEs left over pair arithmetic wins wherever the steps count.  Its setup is the dearer one
// on few nodes and on uniform grids that do not fill the lanes, so few steps of many such PDEs stream,
// and so do many PDEs of few nodes: one to 64 nodes cost it the same.
//
// The terms are fits to measured calls (in ns, 152 SMs), within a fifth of them from 2 to 1000 steps, 8 to
// 2048 nodes and 60 to 131072 PDEs.  Both sides at the lines, ms streaming / pair: 131072 uniform PDEs of 65 nodes, 2
// steps 1.51/2.73, 99 steps (32768) 1.68/1.60; 32768 of 513, 2 steps 3.03/3.56, 29 steps 5.52/4.77; 16384 of 16 nodes, 199
// steps 0.75/0.94, of 32 nodes 1.27/0.89; 131072 of 40, 999 steps 30.7/30.1.
// PDEs left over (a drift across the grid: vol 2 to 5 %, rates of 6 to 10 %) cost pair arithmetic its setup and the FP64
// kernel five times a step, or its latency: ms streaming / pair, all PDEs left over, 99 steps: 32768 of 1024 nodes
// 24.0/50.2, 12000 of them 19.4/18.8; 300 of 512 nodes, 30 of them left over, 255 steps: FP64 on chip 1.19, pair 1.47.
#pragma once

#include <algorithm>
#include <utility>

#include "fd1d_kernels.h"

namespace kwg {

enum class Fp64Route { kPair, kOnChip, kStream };

// A batch by what its cost depends on: PDEs and time steps by padded node count (64, 128, ... 2048).
struct Fp64Batch {
    struct Kind {
        long long n = 0, steps = 0;
        int longest = 0;

        void add(long long count, int s)
        {
            n += count;
            steps += count * s;
            longest = std::max(longest, s);
        }
    };
    struct Cost {
        double sum = 0., longest = 0.;  // throughput, and one PDE's latency

        double ns() const { return std::max(sum, longest); }
    };
    static constexpr int kSizes = 6;
    bool uniform = false;
    Kind plain[kSizes], left[kSizes];
    bool ragged[kSizes] = {};  // a PDE that does not fill the lanes
    long long nodes = 0, node_steps = 0, most_nodes = 0, most_node_steps = 0;

    Fp64Batch() = default;
    explicit Fp64Batch(bool uniform_grid) : uniform(uniform_grid) {}
    // the size class of x nodes
    static int size_of(int x) { return x <= 64 ? 0 : 26 - __builtin_clz((unsigned)x - 1u); }

    // `count` PDEs of x nodes (2048 at most) and s steps, `leaves` of them left over by pair arithmetic
    void add(long long count, int x, int s, long long leaves = 0)
    {
        const int k = size_of(x);
        ragged[k] = ragged[k] || x != 64 << k;
        if (count > leaves) plain[k].add(count - leaves, s);
        if (leaves > 0) left[k].add(leaves, s);
        const long long xs = (long long)x * s;
        nodes += count * x;
        node_steps += count * xs;
        most_nodes = std::max(most_nodes, (long long)x);
        most_node_steps = std::max(most_node_steps, xs);
    }

    void add(const Fp64Batch& o)
    {
        for (int k = 0; k < kSizes; ++k) {
            for (auto [to, from] : {std::pair{&plain[k], &o.plain[k]}, std::pair{&left[k], &o.left[k]}}) {
                to->n += from->n;
                to->steps += from->steps;
                to->longest = std::max(to->longest, from->longest);
            }
            ragged[k] = ragged[k] || o.ragged[k];
        }
        nodes += o.nodes;
        node_steps += o.node_steps;
        most_nodes = std::max(most_nodes, o.most_nodes);
        most_node_steps = std::max(most_node_steps, o.most_node_steps);
    }

    bool any_left() const
    {
        for (const Kind& l : left)
            if (l.n > 0) return true;
        return false;
    }
    double setup_ns(int k) const
    {
        const double n = 64 << k;
        return !uniform ? 20. + 0.145 * n : ragged[k] ? 10. + 0.103 * n : 12. + 0.038 * n;
    }
    // the warp-per-PDE FP64 kernel
    void add_fp64(Cost& c, const Kind& d, int k) const
    {
        constexpr double kStep[kSizes] = {1.45, 2., 3.4, 6., 14.5, 59.};  // 2048 nodes: 64 per lane, spills
        const double n = 64 << k;
        c.sum += 0.16 * n * (double)d.n + (uniform ? 1. : 1.12) * kStep[k] * (double)d.steps;
        c.longest = std::max(c.longest, d.longest * (1200. + 8.8 * n) * (d.n > 304 ? 1.25 : 1.));
    }
    // pair arithmetic; `rest`: of the PDEs it leaves over
    Cost pair(Cost& rest) const
    {
        Cost c;
        long long n_plain = 0, n_all = 0;
        for (int k = 0; k < kSizes; ++k) {
            n_plain += plain[k].n;
            n_all += plain[k].n + left[k].n;
        }
        const double wave = n_plain < 2500 ? 1.5 : 1.;  // a last wave of warps that is mostly empty
        const double warps = n_all <= 304 ? 1. : n_all <= 912 ? 1.4 : 2.2;  // fewer warps per PDE: longer chains
        for (int k = 0; k < kSizes; ++k) {
            const double n = 64 << k, setup = setup_ns(k) * (double)plain[k].n;
            c.sum += wave * std::max(setup, 0.5 * setup + std::max(0.23, 0.0028 * n) * (double)plain[k].steps);
            c.longest = std::max(c.longest, plain[k].longest * (uniform ? 600. + 0.8 * n : 700. + n) *
                                                (k >= 2 && k <= 4 ? warps : 1.));
            rest.sum += setup_ns(k) * (double)left[k].n;
            add_fp64(rest, left[k], k);
        }
        return c;
    }
    Cost on_chip() const
    {
        Cost c;
        for (int k = 0; k < kSizes; ++k) {
            add_fp64(c, plain[k], k);
            add_fp64(c, left[k], k);
        }
        return c;
    }
    double pair_ns() const
    {
        Cost rest;
        const Cost c = pair(rest);
        return c.ns() + rest.ns();
    }
    double on_chip_ns() const { return on_chip().ns(); }
    // One of several batches that run side by side: others fill the time of a few PDEs' chains, so
    // that work counts, not latency.
    bool fp64_beside_others() const
    {
        Cost rest;
        const Cost c = pair(rest);
        return any_left() && on_chip().sum < c.sum + rest.sum;
    }
    Cost stream() const
    {
        int longest = 0;
        for (int k = 0; k < kSizes; ++k) longest = std::max({longest, plain[k].longest, left[k].longest});
        const double x = (double)most_nodes, xs = (double)most_node_steps, s = longest;
        const double all = (double)nodes, all_steps = (double)node_steps;
        if (uniform) return {0.175 * all + 0.0055 * all_steps, 4100. * x + 140. * xs + 1100. * s};
        return {0.33 * all + 0.0078 * all_steps, 7100. * x + 155. * xs + 1250. * s};
    }
    double stream_ns() const { return stream().ns(); }
    // The longest tiles of a streaming launch bind it: they want a scheduler to themselves (one 4-warp block per
    // SM; 131072 PDEs of up to 2048 nodes and 1144 steps, 585 -> 342 ms).
    bool few_long_chains() const
    {
        const Cost c = stream();
        return c.longest > 0.5 * c.sum;
    }
    // FP64 stepping, whichever of the two
    Fp64Route fp64() const { return on_chip_ns() <= stream_ns() ? Fp64Route::kOnChip : Fp64Route::kStream; }
    Fp64Route best() const
    {
        const double p = pair_ns();
        if (any_left() && on_chip_ns() < p && fp64() == Fp64Route::kOnChip) return Fp64Route::kOnChip;
        return stream_ns() < p ? Fp64Route::kStream : Fp64Route::kPair;
    }
};

// FD1D-BS on small grids with few time levels is stepped in FP64: its American and European solve round alike there,
// and the errors cancel to 1e-15 to 6e-15 of the price; pair arithmetic's, which do not, are 3e-15 to 8e-15.  Beyond these
// lines (64 options at scale 5 and 50, 48 to 2048 nodes, 40 to 2048 levels) pair arithmetic is the nearer one.
inline bool bs_in_fp64(int x, int t_dim, bool uniform)
{
    return uniform ? x < 100 && t_dim <= 150 : (x <= 160 && t_dim <= 700) || (x <= 600 && t_dim <= 400);
}

// A batch of m PDEs of x nodes and s steps on the device, where the number left over is known later: from how
// many of them on another solver takes it (m + 1: none), and which.  The cost of pair arithmetic
// grows with that number, the others' do not depend on it.
inline long long pair64_limit(long long m, int x, int s, bool uniform, bool may_stream, Fp64Route* instead)
{
    auto route = [&](long long left) {
        Fp64Batch b(uniform);
        b.add(m, x, s, left);
        if (may_stream) return b.best();
        return left > 0 && b.on_chip_ns() < b.pair_ns() ? Fp64Route::kOnChip : Fp64Route::kPair;
    };
    long long lo = 1, hi = m + 1;
    while (lo < hi) {
        const long long mid = (lo + hi) / 2;
        if (route(mid) != Fp64Route::kPair) hi = mid;
        else lo = mid + 1;
    }
    *instead = lo <= m ? route(lo) : Fp64Route::kPair;
    return lo;
}

}  // namespace kwg
