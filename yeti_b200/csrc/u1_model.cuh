// Host-side preparation of a U1 model (the argument list of
// sys_linmat_lindef_static) into per-patch device arrays, shared by the
// assembly and the shape-gradient kernels.
#pragma once
#include <vector>

#include "common.cuh"

namespace yeti {

struct U1Patch {
    int p[3] = {0, 0, 0};
    int nkv[3] = {0, 0, 0};
    int nn = 0;              // nodes per element
    int nq = 0;              // Gauss points per element (NBINT)
    int ng = 0;              // Gauss points per direction
    double E = 0, nu = 0, rho = 0;
    int64_t elem_begin = 0;  // global index (0-based) of the first element
    int64_t nelem = 0;
    int64_t nactive = 0;
    int64_t nb_data_elem = 0;
    std::vector<int64_t> act;   // global ids (0-based) of active elements
    std::vector<int64_t> slot;  // COO slot offset of each active element
    // views of U1Model::arena
    DevBuf knots;   // U_1 | U_2 | U_3
    DevBuf gauss;   // 4 * nq  (weight, t1, t2, t3)
    DevBuf ien;     // nactive * nn, int32 0-based CP index
    DevBuf w;       // nactive * nn element weights
    DevBuf span;    // nactive * 3, int32 1-based knot span
    DevBuf slotd;   // nactive, int64 slot offsets
    DevBuf gid;     // nactive, int32 global element ids
    // the caller's connectivity and weights of the patch, as they came (owned)
    DevBuf raw_ien, raw_w, conv;
};

struct U1Model {
    DevBuf arena;            // holds the arrays of the patches and coords
    std::vector<U1Patch> patches;
    DevBuf coords;           // 3 * nb_cp
    int64_t nb_cp = 0;
    int64_t nb_data = 0;     // slots needed (sum over active elements)
};

// Validate the model, compute slot offsets (compacted over active
// elements, build_system_elemStorage.f90:156-293) and upload the geometry.
int u1_prepare(yeti_ctx *ctx, const yeti_u1_model *m, U1Model &out);

#ifdef __CUDACC__
// First slot of column node j's blocks, relative to the element's.
__host__ __device__ inline int64_t slot_col(int j) { return 9LL * j * (j - 1) / 2 + 6LL * j; }

// The slots of an element, a warp per column node j (of the nwarp that take
// part) and consecutive lanes on consecutive slots: visit(slot, i, j, row
// component, column component) for the 9 j + 6 slots of the column (9 per node
// i < j with the row component fastest, then the upper triangle of the
// diagonal block).
template <class V>
__device__ __forceinline__ void for_slots(int nn, int64_t base, int warp, int nwarp, V visit) {
    const int lane = threadIdx.x & 31;
    for (int j = warp; j < nn; j += nwarp) {
        const int64_t jb = base + slot_col(j);
        int i = lane / 9, r = lane - 9 * i;
        for (int sl = lane; sl < 9 * j; sl += 32) {
            const int ll = r * 11 >> 5;   // r / 3
            visit(jb + sl, i, j, r - 3 * ll, ll);
            i += 3;                       // 32 = 3 * 9 + 5
            if ((r += 5) >= 9) {
                r -= 9;
                i++;
            }
        }
        if (lane < 6) {
            const int ll = lane < 1 ? 0 : lane < 3 ? 1 : 2;
            visit(jb + 9 * j + lane, j, j, lane - ll * (ll + 1) / 2, ll);
        }
    }
}
#endif

// Element stiffness of one patch's active elements by the sum-factorised
// kernel (stiff_sf.cu), written into the COO slots of the pair kernel.
int launch_u1_stiffness_sf(yeti_ctx *ctx, const U1Patch &P, const double *coords,
                           double lam, double mu, double *kdata, int32_t *krow,
                           int32_t *kcol, size_t smem_cap);

// The distributed and body loads of each element, in order: of(jel) for a
// 1-based element.  As large as the loads' lists of targets and one number per
// element (a mark per load and element would be gigabytes for a thousand loads
// on a million elements).
class ElementLoads {
    struct Node {
        int32_t load, next;
    };
    std::vector<int32_t> head;   // first node of an element, -1: none; empty: no such loads
    std::vector<Node> nodes;

public:
    struct Iter {
        const Node *nodes;
        int32_t i;
        int64_t operator*() const { return nodes[i].load; }
        Iter &operator++() { return i = nodes[i].next, *this; }
        bool operator!=(const Iter &o) const { return i != o.i; }
    };
    struct Range {
        Iter b, e;
        Iter begin() const { return b; }
        Iter end() const { return e; }
    };
    // takes(type): the loads of interest
    template <class F>
    ElementLoads(const yeti_u1_model *m, F takes) {
        int64_t k = 0, targets = 0;
        for (int64_t il = 0; il < m->nb_load; il++) {
            k += m->load_target_nbelem[il];
            if (takes(m->jdltype[il])) targets += m->load_target_nbelem[il];
        }
        if (!targets) return;
        head.assign(m->nb_elem + 1, -1);
        nodes.reserve(targets);
        // from the last load on, each before those that an element has
        for (int64_t il = m->nb_load - 1; il >= 0; il--) {
            const int64_t n = m->load_target_nbelem[il];
            k -= n;
            if (!takes(m->jdltype[il])) continue;
            for (int64_t i = 0; i < n; i++) {
                const int64_t e = m->inddload[k + i];
                if (e < 1 || e > m->nb_elem || (head[e] >= 0 && nodes[head[e]].load == il)) continue;
                nodes.push_back({(int32_t)il, head[e]});
                head[e] = (int32_t)nodes.size() - 1;
            }
        }
    }
    Range of(int64_t jel) const {
        return {{nodes.data(), head.empty() ? -1 : head[jel]}, {nodes.data(), -1}};
    }
};

}  // namespace yeti
