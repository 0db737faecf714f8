// The loads of each element (yeti_b200/csrc/u1_model.cuh) against a scan of the
// loads' target lists, and the memory that building them takes.
#include <cstdio>
#include <cstdlib>
#include <new>
#include <random>
#include <vector>

#include "u1_model.cuh"

static size_t held = 0, peak = 0;
void *operator new(size_t n) {
    size_t *p = static_cast<size_t *>(std::malloc(n + 16));
    *p = n;
    held += n;
    if (held > peak) peak = held;
    return p + 2;
}
void operator delete(void *p) noexcept {
    if (!p) return;
    size_t *q = static_cast<size_t *>(p) - 2;
    held -= *q;
    std::free(q);
}
void operator delete(void *p, size_t) noexcept { operator delete(p); }

#define HOLDS(c)                                                        \
    do {                                                                \
        if (!(c)) {                                                     \
            std::printf("%s:%d: not so: %s\n", __FILE__, __LINE__, #c); \
            std::exit(1);                                               \
        }                                                               \
    } while (0)

static bool takes(int64_t ty) { return ty == 101 || (ty > 9 && ty < 100); }

// nload loads of up to `most` targets, some out of range, repeated or of other types
static void compare(int64_t nelem, int64_t nload, int most, unsigned seed) {
    std::mt19937 rng(seed);
    std::vector<int64_t> ind, type, len;
    for (int64_t il = 0; il < nload; il++) {
        const int64_t types[] = {101, 10, 62, 99, 1, 102, 3};
        type.push_back(types[rng() % 7]);
        len.push_back(rng() % (most + 1));
        for (int64_t i = 0; i < len.back(); i++) ind.push_back((int64_t)(rng() % (nelem + 4)) - 1);
    }
    yeti_u1_model m = {};
    m.nb_elem = nelem;
    m.nb_load = nload;
    m.inddload = ind.data();
    m.jdltype = type.data();
    m.load_target_nbelem = len.data();
    const size_t before = held;
    peak = held;
    const yeti::ElementLoads loads(&m, takes);
    // the lists, and three numbers per element while they are made
    HOLDS(peak - before <= 8 * (ind.size() + 3 * (nelem + 2)));
    for (int64_t e = 1; e <= nelem; e++) {
        std::vector<int64_t> want, got;
        int64_t k = 0;
        for (int64_t il = 0; il < nload; k += len[il++])
            if (takes(type[il]))
                for (int64_t i = 0; i < len[il]; i++)
                    if (ind[k + i] == e) {
                        want.push_back(il);
                        break;
                    }
        for (int64_t il : loads.of(e)) got.push_back(il);
        HOLDS(got == want);
    }
}

int main() {
    compare(1, 0, 0, 1);
    compare(5, 3, 0, 2);
    compare(1, 1, 3, 3);
    compare(40, 30, 60, 4);
    compare(300, 2000, 4, 5);
    compare(4000, 20, 4000, 6);
}
