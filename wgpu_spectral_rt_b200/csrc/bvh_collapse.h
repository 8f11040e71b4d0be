// bvh_collapse.h — which nodes of a binary tree become wide ones.
//
// The cost recurrence of Ylitie, Karras and Laine (HPG 2017, section 3.1):
// cost[i] is the least surface-area cost of a subtree as a forest of at most i
// roots, each a leaf (area x triangles x COLLAPSE_TRI) or a wide node (area x
// COLLAPSE_NODE + its children's forest of `width` roots).  Host and device, so
// that the two functions can be checked over any boxes without a GPU.
//
// Against opening the child of largest area until a node is full, everywhere
// (k_collapse still does at the top): config 2 186k instead of 267k nodes, closest
// hits 3.26 -> 3.22 ms, shadow rays 1.95 -> 1.87; Cornell 640x480 0.73 -> 0.70 and
// 0.47 -> 0.42, photon pass of the animated scene 0.94 -> 0.89.
// Weight of a triangle 0.15 / 0.3 / 0.5 / 0.8 of a node: config 2 closest hits
// 3.29 / 3.26 / 3.26 / 3.24 ms, shadow rays 1.93 / 1.95 / 1.96 / 1.99; animated
// 1.01 / 1.00 / 1.00 / 1.00 and 0.54 / 0.54 / 0.57 / 0.57.
#pragma once

#include <cmath>
#include <cstdint>

#ifdef __CUDACC__
#define SRT_HD __host__ __device__ __forceinline__
#else
#define SRT_HD inline
#endif

namespace srt {

#ifndef SRT_COLLAPSE_TRI
#define SRT_COLLAPSE_TRI 0.3f
#endif
constexpr float COLLAPSE_NODE = 1.0f, COLLAPSE_TRI = SRT_COLLAPSE_TRI;
// Areas are clamped, so that the costs are finite and ordered whatever the
// boxes are (a corner at 1e20 has an infinite area, a NaN one none): the cost of
// 2^30 triangles stays below 1.4e37.  No area is zero: where all boxes are points
// or lines along an axis, every forest would cost the same, wide nodes would get
// two children, and a chain of 40 splits a tree too deep for traversal.
constexpr float COLLAPSE_AREA_MIN = 1e-36f, COLLAPSE_AREA_MAX = 1e28f;

// Half the surface of a box of extents x, y, z, clamped; NaN counts as the least.
SRT_HD float collapse_area(float x, float y, float z) {
    return fminf(fmaxf(x * y + y * z + z * x, COLLAPSE_AREA_MIN), COLLAPSE_AREA_MAX);
}

// From the children's costs l[0..6] and r[0..6] (1 .. 7 roots): the node's
// cost[0..6] and choice[0..7].  choice[i - 1] (i = 2 .. width): roots given to the
// left child, 1 .. i - 1, or (i < width only) 0: the same forest as i - 1 roots;
// choice[0]: 1 if the node alone is a leaf.
SRT_HD void collapse_choose(const float* l, const float* r, float area, uint32_t count, int width, uint32_t leaf_max,
                            float* cost, uint32_t* choice) {
    float best[9];
    uint32_t pick[9] = {0u, 0u, 0u, 0u, 0u, 0u, 0u, 0u, 0u};
#pragma unroll
    for (int i = 2; i <= 8; ++i) {
        // the first split stands unless another costs less, so every pick is one
        best[i] = l[0] + r[i - 2];
        pick[i] = 1u;
#pragma unroll
        for (int k = 2; k < i; ++k) {
            const float c = l[k - 1] + r[i - k - 1];
            if (c < best[i]) {
                best[i] = c;
                pick[i] = (uint32_t)k;
            }
        }
    }
    float wide = best[8];
#pragma unroll
    for (int i = 2; i < 8; ++i)
        if (i == width) wide = best[i];
    best[1] = area * COLLAPSE_NODE + wide;
    choice[0] = 0u;
    if (count <= leaf_max && area * (float)count * COLLAPSE_TRI <= best[1]) {
        best[1] = area * (float)count * COLLAPSE_TRI;
        choice[0] = 1u;
    }
    // the wide node's own distribution is kept even where fewer roots cost as little
#pragma unroll
    for (int i = 2; i <= 8; ++i) {
        choice[i - 1] = pick[i];
        if (i < 8 && i < width && !(best[i] < best[i - 1])) {
            best[i] = best[i - 1];
            choice[i - 1] = 0u;
        }
    }
#pragma unroll
    for (int i = 1; i <= 7; ++i) cost[i - 1] = best[i];
}

// The forest of `width` roots that collapse_choose chose for node `ref`: its
// refs (at most `width`, returned).  TREE: leaf(ref), left(ref), right(ref),
// choice(ref, i).  `ok` is cleared where a choice is out of its range (there is
// none that collapse_choose wrote): that ref stays as it is.
template <class TREE>
SRT_HD int collapse_expand(const TREE& tree, uint32_t ref, int width, uint32_t* refs, bool& ok) {
    int roots[8];  // how many roots refs[c] may become; their sum is at most `width`
    int nc = 1;
    refs[0] = ref;
    roots[0] = width;
    for (int c = 0; c < nc;) {
        if (roots[c] <= 1 || tree.leaf(refs[c])) {
            ++c;
            continue;
        }
        const int k = (int)tree.choice(refs[c], roots[c]);
        if (k == 0) {
            --roots[c];
            continue;
        }
        if (k >= roots[c] || nc >= 8) {
            ok = false;
            ++c;
            continue;
        }
        refs[nc] = tree.right(refs[c]);
        roots[nc++] = roots[c] - k;
        refs[c] = tree.left(refs[c]);
        roots[c] = k;
    }
    return nc;
}

// Slots of a node's nc children, d[c]: the child's centre from the node's.  Slot s
// is visited first by rays whose octant is s (bit set = negative direction), which
// want the child lying farthest along +x/+y/+z for set bits; greedy on the best
// (child, slot) score.  child_in[s]: the child in slot s, or -1.  Every child gets
// a slot of its own whatever the scores are (a box without a centre scores NaN).
SRT_HD void collapse_slots(int nc, const float (*d)[3], int* child_in) {
    uint32_t placed = 0u, taken = 0u;  // children with a slot, slots with a child
    for (int s = 0; s < 8; ++s) child_in[s] = -1;
    for (int it = 0; it < nc; ++it) {
        float bs = -3.4e38f;
        int bc = -1, bsl = -1;
        for (int c = 0; c < nc; ++c) {
            if ((placed >> c) & 1u) continue;
            const float x = d[c][0], y = d[c][1], z = d[c][2];
#pragma unroll
            for (int s = 0; s < 8; ++s) {
                if ((taken >> s) & 1u) continue;
                const float sc = ((s & 1) ? x : -x) + ((s & 2) ? y : -y) + ((s & 4) ? z : -z);
                if (bc < 0 || sc > bs) {
                    bs = sc;
                    bc = c;
                    bsl = s;
                }
            }
        }
        placed |= 1u << bc;
        taken |= 1u << bsl;
        child_in[bsl] = bc;
    }
}

}  // namespace srt
