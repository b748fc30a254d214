// gm_graph_cache.h -- which captured graph serves a solve, and the steps of a
// batch of solves: host logic only, no CUDA, so that its error paths can be
// tested without a GPU (tests/c/test_graph_cache.cpp).
#ifndef GM_GRAPH_CACHE_H
#define GM_GRAPH_CACHE_H

#include <algorithm>
#include <cstddef>
#include <utility>
#include <vector>

namespace gm {

constexpr size_t kGraphCache = 16;  // instantiated graphs kept
// Graphs of one shape that single solves go round, and bindings (10-25 us) that
// cost as much as a capture (1-2 ms).  A batch goes round as many as it has
// images of the shape on a slot.
constexpr int kSameShape = 4, kRebindsPerCapture = 50;

// The graph of a solve: one bound to its buffers already, else one of its
// shape, given its buffers, else a new one.  A program that goes round a few
// sets of buffers gets a graph for each (up to `keep` of them) once the bindings
// have cost as much as a capture.
//
// G has `used` and `rebinds`.  Ops answers for the solve: same_shape(g), bound(g),
// bind(g) and build(g) (0: done) and drop(g), which frees g's graph.  The result
// is valid until the next call.
template <class G, class Ops>
int cached_graph(std::vector<G>& graphs, unsigned long long& clock, int keep, Ops&& ops, G** out)
{
    size_t old = graphs.size();
    int same = 0, rebinds = 0;
    for (size_t i = 0; i < graphs.size(); ++i) {
        G& g = graphs[i];
        if (!ops.same_shape(g)) continue;
        if (ops.bound(g)) {
            g.used = ++clock;
            *out = &g;
            return 0;
        }
        ++same;
        rebinds += g.rebinds;
        if (old == graphs.size() || g.used < graphs[old].used) old = i;
    }
    if (same > 0 && (same >= keep || rebinds < same * kRebindsPerCapture)) {
        G& g = graphs[old];
        if (ops.bind(g) == 0) {
            g.rebinds += 1;
            g.used = ++clock;
            *out = &g;
            return 0;
        }
        // some of its nodes may have the new buffers and the others the old ones
        ops.drop(g);
        graphs.erase(graphs.begin() + (std::ptrdiff_t)old);
    }
    G g = {};
    const int rc = ops.build(g);
    if (rc != 0) return rc;
    g.used = ++clock;
    if (graphs.size() >= kGraphCache) {
        auto lru = std::min_element(graphs.begin(), graphs.end(), [](const G& x, const G& y) { return x.used < y.used; });
        ops.drop(*lru);
        graphs.erase(lru);
    }
    graphs.push_back(std::move(g));
    *out = &graphs.back();
    return 0;
}

// A graph of the solve's shape, whatever it is bound to; in a full cache none is
// captured yet, where it could push out one that is about to be launched.
template <class G, class Ops>
int ready_graph(std::vector<G>& graphs, unsigned long long& clock, int keep, Ops&& ops)
{
    if (graphs.size() >= kGraphCache) return 0;
    for (const G& g : graphs)
        if (ops.same_shape(g)) return 0;
    G* g = nullptr;
    return cached_graph(graphs, clock, keep, ops, &g);
}

// A batch of n solves on several streams.  Ops: ready(k), solve k has a graph;
// begin(), the streams follow the caller's; launch(k); join(), the caller's stream
// follows them and has been waited for (0: done).  A solve in flight writes the
// caller's vectors and uses its slot's workspace, so after a failure it is
// waited for (drain()) before the error is returned; *launched tells a failure
// that came before any launch, after which another way may be tried.
template <class Ops>
int run_images(int n, Ops&& ops, bool* launched)
{
    *launched = false;
    for (int k = 0; k < n; ++k)
        if (const int rc = ops.ready(k)) return rc;
    int rc = ops.begin();
    if (rc != 0) return rc;
    for (int k = 0; k < n && rc == 0; ++k) {
        *launched = true;
        rc = ops.launch(k);
    }
    if (rc == 0) rc = ops.join();
    if (rc != 0) ops.drain();
    return rc;
}

}  // namespace gm

#endif
