"""The functions that pick the wide tree's nodes (bvh_collapse.h), compiled for
the host: over boxes of any size, infinite and NaN ones included, every choice
is a split of its roots, no node gets more than `width` children, the wide
nodes cover every leaf exactly once, and every child has a slot of its own."""
from __future__ import annotations

import ctypes as C
import subprocess

import numpy as np
import pytest

from conftest import ROOT

SOURCE = r"""
#include <cmath>
#include <cstdint>
#include <stdexcept>
#include <vector>
#include "bvh_collapse.h"
using namespace srt;
namespace {
constexpr uint32_t LEAF = 0x80000000u;
struct Box { float lo[3], hi[3]; };
struct Tree {
    std::vector<uint32_t> l, r, n;
    std::vector<Box> box;
    std::vector<std::vector<uint32_t>> ch;
    const float* leaves;
    mutable long calls = 0;
    bool leaf(uint32_t ref) const { return (ref & LEAF) != 0; }
    uint32_t left(uint32_t ref) const { return l.at(ref); }
    uint32_t right(uint32_t ref) const { return r.at(ref); }
    uint32_t choice(uint32_t ref, int i) const {
        if (i < 1 || i > 8 || ++calls > 1000000) throw std::out_of_range("choice");
        return ch.at(ref)[i - 1];
    }
};
Box box_of(const Tree& t, uint32_t ref) {
    if (!t.leaf(ref)) return t.box[ref];
    Box b;
    for (int a = 0; a < 3; ++a) b.lo[a] = t.leaves[6 * (ref & ~LEAF) + a], b.hi[a] = t.leaves[6 * (ref & ~LEAF) + 3 + a];
    return b;
}
float area_of(const Box& b) { return collapse_area(b.hi[0] - b.lo[0], b.hi[1] - b.lo[1], b.hi[2] - b.lo[2]); }
// split: 0 the middle, 1 one leaf on the right (a chain)
uint32_t make(Tree& t, uint32_t first, uint32_t count, int split, int width, uint32_t leaf_max, std::vector<float>& cost) {
    cost.resize(7);
    if (count == 1) {
        const float c = area_of(box_of(t, LEAF | first)) * COLLAPSE_TRI;
        for (float& x : cost) x = c;
        return LEAF | first;
    }
    const uint32_t id = (uint32_t)t.l.size(), left = split ? count - 1 : count / 2;
    t.l.push_back(0), t.r.push_back(0), t.n.push_back(count), t.box.emplace_back(), t.ch.emplace_back(8);
    std::vector<float> cl, cr;
    const uint32_t a = make(t, first, left, split, width, leaf_max, cl);
    const uint32_t b = make(t, first + left, count - left, split, width, leaf_max, cr);
    t.l[id] = a, t.r[id] = b;
    const Box x = box_of(t, a), y = box_of(t, b);
    for (int k = 0; k < 3; ++k) t.box[id].lo[k] = fminf(x.lo[k], y.lo[k]), t.box[id].hi[k] = fmaxf(x.hi[k], y.hi[k]);
    collapse_choose(cl.data(), cr.data(), area_of(t.box[id]), count, width, leaf_max, cost.data(), t.ch[id].data());
    for (int i = 2; i <= width; ++i)
        if (t.ch[id][i - 1] >= (uint32_t)i || (i == width && t.ch[id][i - 1] == 0)) throw std::logic_error("choice");
    for (float c : cost)
        if (!std::isfinite(c)) throw std::logic_error("cost");
    return id;
}
}  // namespace
// out: wide nodes, their levels, children over all, leaves covered; returns 0, or what failed
extern "C" int collapse_tree(const float* leaves, uint32_t n, int split, int width, uint32_t leaf_max, uint32_t* seen,
                             uint32_t* out) {
    try {
        Tree t;
        t.leaves = leaves;
        std::vector<float> cost;
        std::vector<uint32_t> level{make(t, 0, n, split, width, leaf_max, cost)}, next;
        out[0] = out[1] = out[2] = 0;
        for (; !level.empty(); level.swap(next), next.clear()) {
            ++out[1];
            for (uint32_t ref : level) {
                uint32_t refs[8];
                bool ok = true;
                const int nc = collapse_expand(t, ref, width, refs, ok);
                if (!ok) return 1;
                if (nc < 2 || nc > width) return 2;
                ++out[0];
                out[2] += nc;
                for (int c = 0; c < nc; ++c) {
                    if (t.leaf(refs[c])) ++seen[refs[c] & ~LEAF];
                    else if (t.n[refs[c]] <= leaf_max && t.choice(refs[c], 1)) {
                        std::vector<uint32_t> below{refs[c]};
                        while (!below.empty()) {
                            const uint32_t q = below.back();
                            below.pop_back();
                            if (t.leaf(q)) ++seen[q & ~LEAF];
                            else below.push_back(t.l[q]), below.push_back(t.r[q]);
                        }
                    } else next.push_back(refs[c]);
                }
            }
        }
        return 0;
    } catch (const std::out_of_range&) { return 3; } catch (const std::logic_error&) { return 4; }
}
extern "C" void slots(int nc, const float* d, int* child_in) { collapse_slots(nc, (const float (*)[3])d, child_in); }
"""


@pytest.fixture(scope="module")
def library(tmp_path_factory):
    d = tmp_path_factory.mktemp("collapse")
    (d / "collapse.cpp").write_text(SOURCE)
    subprocess.run(["g++", "-O1", "-std=c++17", "-fPIC", "-shared", f"-I{ROOT}/wgpu_spectral_rt_b200/csrc",
                    str(d / "collapse.cpp"), "-o", str(d / "collapse.so")], check=True, timeout=120)
    return C.CDLL(str(d / "collapse.so"))


@pytest.fixture(scope="module")
def collapse(library):
    fn = library.collapse_tree

    def run(boxes, split=0, width=8, leaf_max=2):
        n = len(boxes)
        seen, out = np.zeros(n, np.uint32), np.zeros(3, np.uint32)
        p = [np.ascontiguousarray(x).ctypes.data_as(C.c_void_p) for x in (boxes, seen, out)]
        err = fn(p[0], n, split, width, leaf_max, p[1], p[2])
        return err, seen, out

    return run


def _boxes(n, seed=1):
    g = np.random.default_rng(seed)
    c = np.sort(g.uniform(-1, 1, n)).astype(np.float32)
    b = np.zeros((n, 6), np.float32)
    b[:, 0] = c
    b[:, 1:3] = g.uniform(-1, 1, (n, 2))
    b[:, 3:] = b[:, :3] + g.uniform(0.001, 0.05, (n, 3)).astype(np.float32)
    return b


@pytest.mark.parametrize("width", [8, 5, 2])
@pytest.mark.parametrize("split", [0, 1])
@pytest.mark.parametrize("extent", [1.0, 1e13, 1e14, 1e18, 1e19, 1e20, 3.3e38, np.inf, np.nan])
def test_any_extent_gives_a_whole_tree(collapse, extent, split, width):
    boxes = _boxes(600)
    if not np.isnan(extent):
        boxes[200, :3], boxes[200, 3:] = -extent, extent
        boxes[201, 4] = extent
    else:
        boxes[200] = np.nan
        boxes[300, 1] = np.nan
    err, seen, out = collapse(boxes, split, width)
    assert err == 0
    assert np.all(seen == 1)
    assert out[2] <= width * out[0]


def test_all_boxes_beyond_the_largest_area(collapse):
    boxes = _boxes(600)
    boxes[:, :3], boxes[:, 3:] = -2e19, 2e19
    err, seen, out = collapse(boxes)
    assert err == 0 and np.all(seen == 1)
    assert out[1] <= 6  # full nodes: 8^4 > 600 leaves


@pytest.mark.parametrize("value", [0.0, 1.0, 3e38, -3.4e38, np.inf, -np.inf, np.nan])
@pytest.mark.parametrize("nc", [1, 2, 7, 8])
def test_every_child_gets_a_slot_of_its_own(library, nc, value):
    for where in ("one", "axis", "all"):
        d = np.random.default_rng(nc).normal(size=(8, 3)).astype(np.float32)
        if where == "one":
            d[nc - 1] = value
        elif where == "axis":
            d[:, 1] = value
        else:
            d[:] = value
        child_in = np.zeros(8, np.int32)
        library.slots(nc, d.ctypes.data_as(C.c_void_p), child_in.ctypes.data_as(C.c_void_p))
        assert sorted(child_in[child_in >= 0]) == list(range(nc))
        assert np.count_nonzero(child_in < 0) == 8 - nc


@pytest.mark.parametrize("kind", ["points", "line", "tiny"])
def test_boxes_without_area_fill_their_nodes(collapse, kind):
    boxes = np.zeros((200, 6), np.float32)
    if kind == "line":
        boxes[:, 0] = np.arange(200)
        boxes[:, 3] = boxes[:, 0] + 0.5
    elif kind == "tiny":
        boxes = _boxes(200) * np.float32(1e-24)
    for split, levels in ((0, 3), (1, 30)):  # 8^3 > 200; 7 more leaves per node of a chain, as it is opened from its end
        err, seen, out = collapse(boxes, split)
        assert err == 0 and np.all(seen == 1)
        assert out[1] <= levels
