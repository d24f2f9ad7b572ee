/* Runs the component labels' steps (csrc/l3d_labels.h) as concurrent threads on the host: every access to
 * a label hands control to a scheduler, which lets a random thread make the next one. */
#include <ucontext.h>

#include <random>
#include <vector>

#include "l3d_labels.h"

namespace {

struct Run {
    std::vector<uint32_t> label;
    std::mt19937 rng;
    ucontext_t main_context;
    struct Thread {
        ucontext_t context;
        std::vector<char> stack;
        bool done = false;
    };
    std::vector<Thread> threads;
    int current = 0, err = 0;
    void (*body)(Run&, uint32_t) = nullptr;
    const uint32_t* edges = nullptr;

    void yield() { swapcontext(&threads[current].context, &main_context); }
    uint32_t load(uint32_t v) { yield(); return label[v]; }
    void store(uint32_t v, uint32_t l) { yield(); label[v] = l; }
    bool swap(uint32_t v, uint32_t from, uint32_t to) {
        yield();
        if (label[v] != from) return false;
        label[v] = to;
        return true;
    }

    static void enter(unsigned lo, unsigned hi, unsigned i) {
        Run& r = *(Run*)((size_t)hi << 32 | lo);
        r.body(r, i);
        r.threads[i].done = true;
        swapcontext(&r.threads[i].context, &r.main_context);
    }
    void all(uint32_t n, void (*f)(Run&, uint32_t)) {
        body = f;
        threads.resize(n);
        std::vector<int> open;
        for (uint32_t i = 0; i < n; i++) {
            Thread& t = threads[i];
            t.stack.resize(16384);
            t.done = false;
            getcontext(&t.context);
            t.context.uc_stack.ss_sp = t.stack.data();
            t.context.uc_stack.ss_size = t.stack.size();
            t.context.uc_link = nullptr;
            const size_t self = (size_t)this;
            makecontext(&t.context, (void (*)())enter, 3, (unsigned)self, (unsigned)(self >> 32), i);
            open.push_back((int)i);
        }
        while (!open.empty()) {
            const size_t k = rng() % open.size();
            current = open[k];
            swapcontext(&main_context, &threads[current].context);
            if (threads[current].done) {
                open[k] = open.back();
                open.pop_back();
            }
        }
    }
};

}  // namespace

/* One run over n vertices: `label` as it stands is flattened, or (edges given) the edges are joined first,
 * a thread per edge.  Returns the error flag. */
extern "C" int label_orders(uint32_t n, uint32_t* label, uint32_t n_edges, const uint32_t* edges, uint32_t seed) {
    Run r;
    r.rng.seed(seed);
    r.label.assign(label, label + n);
    r.edges = edges;
    if (n_edges)
        r.all(n_edges, [](Run& q, uint32_t i) { l3d_label_unite(q, q.edges[2 * i], q.edges[2 * i + 1], &q.err); });
    r.all(n, [](Run& q, uint32_t v) { l3d_label_flatten(q, v, &q.err); });
    for (uint32_t v = 0; v < n; v++) label[v] = r.label[v];
    return r.err;
}

extern "C" uint32_t label_rank(uint32_t v) { return l3d_label_rank(v); }
