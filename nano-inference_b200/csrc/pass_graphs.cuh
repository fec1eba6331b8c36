// Captured launch sequences by kind, for host code.
#pragma once
#include <cstddef>
#include <map>

namespace mi {

// The first pass of a kind runs plainly, the second is captured, later ones replay.  Capturing and instantiating takes 3 - 28 ms
// (36 layers), so what is used stays: where there is no room, the graph used longest ago leaves, by itself, and its kind starts over.  A server
// that decodes 1 .. 64 sequences at a time in two attention ranges has 128 kinds; their graphs hold 143 MB of device memory at 36 layers.
template <class Key, size_t MaxGraphs = 128, size_t MaxKinds = 512>
class PassGraphs {
    struct Entry { void* graph = nullptr; unsigned long long used = 0; };
    std::map<Key, Entry> kinds;
    size_t n_graphs = 0;
    unsigned long long clock = 0;

    // the least recently used kind other than `keep`, among those with a graph or among all
    typename std::map<Key, Entry>::iterator oldest(const Key* keep, bool with_graph) {
        auto o = kinds.end();
        for (auto i = kinds.begin(); i != kinds.end(); ++i)
            if ((!with_graph || i->second.graph) && !(keep && !(i->first < *keep) && !(*keep < i->first)) && (o == kinds.end() || i->second.used < o->second.used)) o = i;
        return o;
    }
    template <class Destroy>
    void erase(typename std::map<Key, Entry>::iterator i, Destroy destroy) {
        if (i->second.graph) { destroy(i->second.graph); n_graphs--; }
        kinds.erase(i);
    }

public:
    // A pass of this kind is about to run.  Returns its graph, or null; *again: it has run before, so it is worth capturing.
    template <class Destroy>
    void* use(const Key& k, bool* again, Destroy destroy) {
        auto i = kinds.find(k);
        *again = i != kinds.end();
        if (!*again) {
            if (kinds.size() >= MaxKinds) erase(oldest(nullptr, false), destroy);
            i = kinds.emplace(k, Entry{}).first;
        }
        i->second.used = ++clock;
        return i->second.graph;
    }
    // the graph of the kind that has just been passed to use()
    template <class Destroy>
    void put(const Key& k, void* graph, Destroy destroy) {
        if (n_graphs >= MaxGraphs) erase(oldest(&k, true), destroy);
        Entry& e = kinds[k];
        if (e.graph) destroy(e.graph); else n_graphs++;
        e.graph = graph;
    }
    // what the graphs point into is about to go; the kinds stay known
    template <class Destroy>
    void drop_graphs(Destroy destroy) {
        for (auto& k : kinds) if (k.second.graph) { destroy(k.second.graph); k.second.graph = nullptr; }
        n_graphs = 0;
    }
    size_t graphs() const { return n_graphs; }
    size_t size() const { return kinds.size(); }
};

}  // namespace mi
