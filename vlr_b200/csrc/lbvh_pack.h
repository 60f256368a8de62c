// Depth-first placement of a hierarchy's nodes and leaves, and the checks that
// make the packed arrays safe to walk.  Plain C++ so that the host can run it
// over hierarchies no build produces.
#pragma once

#include "core.cuh"

namespace vlrb {

// Where node i and its children go.
struct PackedNode {
    uint32_t place, firstLeaf, leaf1;   // its place, and the places of its children's first leaves
    int child0, child1;                 // references in the packed order (~leaf for a leaf)
};

// A node's first child follows it, the second child follows the first's
// subtree; both places and the place of the node's first leaf among the
// leaves are summed on the way up to the root.  `count`: leaves below every
// internal node.  Returns false unless the node's references and its way up
// are those of a tree: both children in range and recorded under this node
// alone, the way ending at node 0, which has no parent, and places in range.
// When that holds for all nodes the references form one tree over the n
// leaves (each node but the root is the child of exactly one, and none hangs
// from a cycle), so a descent from the root ends.
VLRB_HD bool placeNode(const int32_t* children, const int32_t* parentOfNode, const int32_t* parentOfLeaf,
                       const uint32_t* count, uint32_t n, uint32_t i, PackedNode* out) {
    const int last = static_cast<int>(n) - 1;
    const int self = static_cast<int>(i);
    const int c0 = children[2 * i], c1 = children[2 * i + 1];
    if (c0 >= last || c1 >= last || ~c0 > last || ~c1 > last || c0 == c1) return false;
    if ((c0 >= 0 ? parentOfNode[c0] : parentOfLeaf[~c0]) != self) return false;
    if ((c1 >= 0 ? parentOfNode[c1] : parentOfLeaf[~c1]) != self) return false;
    uint32_t place = 0, firstLeaf = 0, steps = 0;
    int node = self, up = parentOfNode[node];
    for (; up >= 0 && up < last && steps < n; up = parentOfNode[node], ++steps) {
        const int left = children[2 * up];
        place += 1;
        if (left != node) {
            const uint32_t leaves = left >= 0 && left < last ? count[left] : 1u;
            place += leaves - 1;
            firstLeaf += leaves;
        }
        node = up;
    }
    if (up >= 0 || node != 0) return false;
    const uint32_t leaves0 = c0 >= 0 ? count[c0] : 1u;
    out->place = place;
    out->firstLeaf = firstLeaf;
    out->leaf1 = firstLeaf + leaves0;
    const uint32_t node0 = place + 1, node1 = place + leaves0;
    if (leaves0 == 0 || place >= n - 1 || out->leaf1 >= n || (c0 >= 0 && node0 >= n - 1) || (c1 >= 0 && node1 >= n - 1))
        return false;
    out->child0 = c0 >= 0 ? static_cast<int>(node0) : ~static_cast<int>(firstLeaf);
    out->child1 = c1 >= 0 ? static_cast<int>(node1) : ~static_cast<int>(out->leaf1);
    return true;
}

} // namespace vlrb
