// Binned-SAH build of a binary tree on the host.
#pragma once

#include <cstddef>
#include <cstdint>
#include <initializer_list>

#include <vector_types.h>

namespace gbsp {

constexpr uint32_t kBinLeaf = 0x80000000u;  // child reference of a binary tree: a primitive

// A binary tree over n >= 2 primitives in the form the collapse reads:
// internal nodes 0 .. n-2 (root 0), child references with kBinLeaf for a
// primitive (its sorted position), each internal node's range [first, last]
// of sorted positions and its box, order[sorted position] = primitive, and the
// primitives' boxes.  The constructor lays it out in one block of size(n)
// float4, on the host or on the device, so that it moves in one copy.
template <class F4, class U4>
struct BinaryTree {
    F4 *primLo, *primHi, *nodeLo, *nodeHi;
    U4 *left, *right, *first, *last, *order;

    BinaryTree() = default;
    BinaryTree(F4 *base, uint32_t n)
    {
        primLo = base, primHi = primLo + n, nodeLo = primHi + n, nodeHi = nodeLo + n;
        F4 *p = nodeHi + n;
        for (U4 **a : {&left, &right, &first, &last, &order}) {
            *a = reinterpret_cast<U4 *>(p);
            p += words(n);
        }
    }
    static size_t words(uint32_t n) { return ((size_t)n + 3) / 4; }
    static size_t size(uint32_t n) { return 4 * (size_t)n + 5 * words(n); }
};

// Top-down binned SAH build (Wald, "On fast construction of SAH-based
// bounding volume hierarchies", 2007) over n >= 2 primitive boxes (w lanes
// zero), split down to single primitives: at every node the primitives'
// centroids are binned into 64 slabs along each axis, and the split between
// bins that minimises area(left) x count(left) + area(right) x count(right)
// partitions the node's range (a median split when every centroid
// coincides).  Node boxes are exact unions.
void sah_binary_tree(const float4 *lo, const float4 *hi, uint32_t n,
    const BinaryTree<float4, uint32_t> &tree);

}  // namespace gbsp
