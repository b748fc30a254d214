// The cache of captured solves (csrc/gm_graph_cache.h) with a fake capture: a
// graph has ten nodes, each with the buffer it was given last, and setting a
// node can be made to fail.  And the steps of a batch with one that fails.
#include <algorithm>
#include <cstdio>
#include <cstdlib>
#include <vector>

#include "gm_graph_cache.h"

#define CHECK(c) \
    do { \
        if (!(c)) { \
            std::printf("line %d: %s\n", __LINE__, #c); \
            std::exit(1); \
        } \
    } while (0)

constexpr int kNodes = 10;
static int g_alive = 0, g_builds = 0, g_sets = 0, g_fail_at = -1;  // g_fail_at: the node that cannot be set

struct Graph {
    int shape, key, node[kNodes];
    unsigned long long used;
    int rebinds;
};

struct Solve {
    int shape, buffer;
    bool build_fails = false;
    bool same_shape(const Graph& g) const { return g.shape == shape; }
    bool bound(const Graph& g) const { return g.key == buffer; }
    int bind(Graph& g) const
    {
        for (int i = 0; i < kNodes; ++i) {
            if (i == g_fail_at) return 2;
            g.node[i] = buffer;
            ++g_sets;
        }
        g.key = buffer;
        return 0;
    }
    int build(Graph& g) const
    {
        if (build_fails) return 2;
        g.shape = shape;
        g.key = buffer;
        for (int& n : g.node) n = buffer;
        ++g_alive;
        ++g_builds;
        return 0;
    }
    void drop(Graph&) const { --g_alive; }
};

struct Cache {
    std::vector<Graph> graphs;
    unsigned long long clock = 0;
    // The buffers the solve's launch would use; -1: no graph.
    bool launch(int shape, int buffer, bool build_fails = false)
    {
        Graph* g = nullptr;
        if (gm::cached_graph(graphs, clock, gm::kSameShape, Solve{shape, buffer, build_fails}, &g) != 0) return false;
        CHECK(g != nullptr && g->shape == shape);
        for (int n : g->node) CHECK(n == buffer);
        CHECK((int)graphs.size() == g_alive && graphs.size() <= gm::kGraphCache);
        return true;
    }
    ~Cache() { g_alive -= (int)graphs.size(); }
};

// A binding that fails half-way, at every node: the solve gets a graph of its
// own, and none that mixes two solves' buffers is left for the first one.
static void failing_bind()
{
    for (int at = 0; at < kNodes; ++at)
        for (int again = 0; again < 2; ++again) {
            Cache c;
            CHECK(c.launch(1, 100));
            g_fail_at = at;
            CHECK(c.launch(1, 200));
            g_fail_at = -1;
            CHECK(c.launch(1, 100));
            CHECK(c.launch(1, 200));
            // and where the capture that takes its place fails too
            g_fail_at = at;
            CHECK(!c.launch(1, 300, true));
            g_fail_at = -1;
            CHECK(c.launch(1, again ? 100 : 200));
            CHECK(c.launch(1, again ? 200 : 100));
            CHECK((int)c.graphs.size() == g_alive);
        }
    CHECK(g_alive == 0);
}

// Shapes past the cache's size, and buffers in turn: every launch has its own.
static void many_shapes()
{
    Cache c;
    for (int i = 0; i < 2000; ++i) CHECK(c.launch(i % 23, i % 7));
    CHECK((int)c.graphs.size() == (int)gm::kGraphCache);
}

// A repeated batch with n images of one shape on a slot: at most one binding an
// image and call, and none once each has a graph of its own, where the cache
// holds that many.
static void repeated_batch()
{
    for (int n = 1; n <= 20; ++n) {
        Cache c;
        const int keep = std::min(n, (int)gm::kGraphCache), builds = g_builds;
        int sets = 0;
        for (int call = 0; call < 1000; ++call) {
            const int before = g_sets;
            for (int k = 0; k < n; ++k) CHECK(gm::ready_graph(c.graphs, c.clock, keep, Solve{1, k}) == 0);
            CHECK(g_sets == before);
            for (int k = 0; k < n; ++k) {
                Graph* g = nullptr;
                CHECK(gm::cached_graph(c.graphs, c.clock, keep, Solve{1, k}, &g) == 0 && g->key == k);
            }
            sets = g_sets - before;
            CHECK(sets <= n * kNodes);
        }
        CHECK(n > keep || sets == 0);
        CHECK(g_builds - builds <= (int)gm::kGraphCache);
    }
    // images of n shapes each: at most one capture an image and call
    for (int n = 1; n <= 40; ++n) {
        Cache c;
        for (int call = 0; call < 5; ++call) {
            const int before = g_builds;
            for (int k = 0; k < n; ++k) CHECK(gm::ready_graph(c.graphs, c.clock, 1, Solve{k, k}) == 0);
            for (int k = 0; k < n; ++k) CHECK(c.launch(k, k));
            CHECK(g_builds - before <= (call > 0 && n <= (int)gm::kGraphCache ? 0 : n));
        }
    }
}

// A batch whose step number `fail_at` fails: nothing is left in flight, and a
// failure counts as one before the launches only where nothing was launched.
struct Batch {
    int n, fail_at;
    int step = 0, launches = 0, in_flight = 0;
    int next() { return step++ == fail_at ? 7 : 0; }
    int ready(int) { return next(); }
    int begin() { return next(); }
    int launch(int)
    {
        ++launches;
        ++in_flight;  // also where the call that follows the launch fails
        return next();
    }
    int join()
    {
        const int rc = next();
        if (rc == 0) in_flight = 0;
        return rc;
    }
    void drain() { in_flight = 0; }
};

static void failing_batch()
{
    for (int n = 1; n < 5; ++n)
        for (int at = -1; at < 2 * n + 2; ++at) {
            Batch b{n, at};
            bool launched = false;
            const int rc = gm::run_images(n, b, &launched);
            CHECK(rc == (at < 0 ? 0 : 7));
            CHECK(b.in_flight == 0);
            CHECK(launched == (b.launches > 0));
            CHECK(at < 0 ? b.launches == n : b.launches <= n);
        }
}

int main()
{
    failing_bind();
    many_shapes();
    repeated_batch();
    failing_batch();
    std::printf("Test PASSED\n");
    return 0;
}
