"""The traversal's packed hierarchy on the CPU: the placement and checks the
packing kernel runs (csrc/lbvh_pack.h), over every array of child references
of small hierarchies, most of them no tree at all."""
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

SRC = r"""
#include "lbvh_pack.h"
#include <cstdio>
#include <vector>
using namespace vlrb;

// parents and leaf counts as the build's kernels make them, one leaf after another
static bool pack(const std::vector<int32_t> &ch, uint32_t n, std::vector<PackedNode> *slots, std::vector<char> *set) {
    const int last = int(n) - 1;
    std::vector<int32_t> pn(n, -1), pl(n, -1);
    for (int i = 0; i < last; ++i)
        for (int k = 0; k < 2; ++k) {
            const int c = ch[2 * i + k];
            if (c >= 0 && c < last) pn[c] = i;
            else if (c < 0 && ~c < int(n)) pl[~c] = i;
        }
    pn[0] = -1;
    std::vector<uint32_t> arrivals(n, 0), count(n, 0);
    for (uint32_t leaf = 0; leaf < n; ++leaf)
        for (int node = pl[leaf]; node >= 0 && node < last; node = pn[node]) {
            if (arrivals[node]++ != 1u) break;
            uint32_t c = 0;
            for (int k = 0; k < 2; ++k) {
                const int x = ch[2 * node + k];
                c += x >= 0 && x < last ? count[x] : 1u;
            }
            count[node] = c;
        }
    bool all = true;
    slots->assign(n, PackedNode{ 0, 0, 0, ~0, ~0 });
    set->assign(n, 0);
    for (uint32_t i = 0; i + 1 < n; ++i) {
        PackedNode p;
        if (!placeNode(ch.data(), pn.data(), pl.data(), count.data(), n, i, &p)) { all = false; continue; }
        if (p.place + 1 >= n || p.leaf1 >= n) return std::printf("place out of range\n"), false;
        (*slots)[p.place] = p;
        (*set)[p.place] = 1;
    }
    return all;
}

// is it a tree over its n leaves, by walking it
static bool isTree(const std::vector<int32_t> &ch, uint32_t n) {
    std::vector<char> seenNode(n, 0), seenLeaf(n, 0);
    std::vector<int> stack{ 0 };
    uint32_t nodes = 0, leaves = 0;
    while (!stack.empty()) {
        const int x = stack.back();
        stack.pop_back();
        if (x >= 0) {
            if (x >= int(n) - 1 || seenNode[x]) return false;
            seenNode[x] = 1;
            ++nodes;
            stack.push_back(ch[2 * x]);
            stack.push_back(ch[2 * x + 1]);
        }
        else {
            if (~x >= int(n) || seenLeaf[~x]) return false;
            seenLeaf[~x] = 1;
            ++leaves;
        }
    }
    return nodes == n - 1 && leaves == n;
}

int main() {
    for (uint32_t n = 2; n <= 4; ++n) {
        // references from one below the last leaf to one above the last node
        const int lo = -int(n) - 1, hi = int(n) - 1, values = hi - lo + 1, refs = 2 * (int(n) - 1);
        long total = 1, trees = 0, accepted = 0;
        for (int i = 0; i < refs; ++i) total *= values;
        for (long code = 0; code < total; ++code) {
            std::vector<int32_t> ch(refs);
            long c = code;
            for (int i = 0; i < refs; ++i) { ch[i] = lo + int(c % values); c /= values; }
            std::vector<PackedNode> slots;
            std::vector<char> set;
            const bool ok = pack(ch, n, &slots, &set), tree = isTree(ch, n);
            trees += tree;
            accepted += ok;
            if (ok != tree) return std::printf("n %u code %ld: accepted %d, tree %d\n", n, code, ok, tree), 1;
            if (!ok) continue;
            // the packed references: every node and leaf met once, in order
            std::vector<int> stack{ 0 };
            uint32_t nextNode = 0, nextLeaf = 0;
            while (!stack.empty()) {
                const int x = stack.back();
                stack.pop_back();
                if (x < 0) { if (uint32_t(~x) != nextLeaf++) return std::printf("leaf order, code %ld\n", code), 1; continue; }
                if (uint32_t(x) != nextNode++ || !set[x]) return std::printf("node order, code %ld\n", code), 1;
                stack.push_back(slots[x].child1);
                stack.push_back(slots[x].child0);
            }
            if (nextNode != n - 1 || nextLeaf != n) return std::printf("incomplete, code %ld\n", code), 1;
        }
        std::printf("%u: %ld arrays, %ld trees, %ld accepted\n", n, total, trees, accepted);
    }
    return 0;
}
"""


def test_only_trees_are_packed_and_each_packed_tree_is_complete(tmp_path):
    src, exe = tmp_path / "pack.cpp", tmp_path / "pack"
    src.write_text(SRC)
    subprocess.run(["g++", "-std=c++17", "-O2", "-I", os.path.join(ROOT, "vlr_b200", "csrc"), str(src), "-o", str(exe)],
                   check=True)
    p = subprocess.run([str(exe)], capture_output=True, text=True, timeout=300)
    assert p.returncode == 0, p.stdout
    assert p.stdout.count("trees") == 3
