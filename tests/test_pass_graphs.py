"""The captured passes of a model (csrc/pass_graphs.cuh), compiled for the host: a kind is captured at its second use and once, as long as it
is used more recently than others there is room for; graphs and kinds are bounded; every graph is destroyed once."""
import subprocess
from pathlib import Path

SRC = Path(__file__).resolve().parent.parent / "nano-inference_b200" / "csrc"

PROGRAM = r"""
#include "pass_graphs.cuh"
#include <cstdio>
#include <cstdlib>
#include <random>
#include <set>
#include <utility>

#define CHECK(c) do { if (!(c)) { std::printf("line %d: %s\n", __LINE__, #c); return 1; } } while (0)
using Key = std::pair<int, int>;
static std::set<void*> live;
static long made = 0;
static void destroy(void* g) { if (!live.erase(g)) { std::printf("destroyed twice\n"); std::exit(1); } std::free(g); }
// one pass; what it did: 0 plain, 1 captured, 2 replayed
template <class G> static int pass(G& g, Key k) {
    bool again;
    if (g.use(k, &again, destroy)) return 2;
    if (!again) return 0;
    void* x = std::malloc(1);
    live.insert(x); made++;
    g.put(k, x, destroy);
    return 1;
}
int main() {
    {   // sequences come and go, 1 .. 64 of them, in two attention ranges: nothing is captured twice
        mi::PassGraphs<Key> g;
        std::mt19937 rng(1);
        int n = 32; made = 0;
        for (int i = 0; i < 100000; i++) {
            n = n + (int)(rng() % 3) - 1; n = n < 1 ? 1 : n > 64 ? 64 : n;
            pass(g, {n, (int)(rng() % 2)});
        }
        CHECK(made <= 128 && g.graphs() == live.size() && g.size() <= 128);
        g.drop_graphs(destroy);
        CHECK(live.empty() && g.graphs() == 0);
        CHECK(pass(g, {32, 0}) == 1);                       // the kinds stay known
        g.drop_graphs(destroy);
    }
    {   // no room: the longest unused graph leaves, the others stay
        mi::PassGraphs<Key, 4, 6> g;
        for (int k = 0; k < 4; k++) { CHECK(pass(g, {k, 0}) == 0); CHECK(pass(g, {k, 0}) == 1); CHECK(pass(g, {k, 0}) == 2); }
        CHECK(pass(g, {0, 0}) == 2);                         // 1 is the oldest now
        CHECK(pass(g, {4, 0}) == 0 && pass(g, {4, 0}) == 1 && g.graphs() == 4);
        for (int k : {0, 2, 3, 4}) CHECK(pass(g, {k, 0}) == 2);
        CHECK(pass(g, {1, 0}) == 0);                         // starts over
        for (int k = 10; k < 100; k++) { CHECK(pass(g, {k, 0}) == 0); CHECK(g.size() <= 6 && g.graphs() <= 4 && g.graphs() == live.size()); }
        g.drop_graphs(destroy);
        CHECK(live.empty());
    }
    return 0;
}
"""


def test_the_least_recently_used_graph_leaves(tmp_path):
    src = tmp_path / "graphs.cpp"
    src.write_text(PROGRAM)
    exe = tmp_path / "graphs"
    subprocess.run(["g++", "-O2", "-Wall", "-std=c++17", "-I", str(SRC), "-o", str(exe), str(src)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout
