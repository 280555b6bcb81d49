"""The tree's builder on geometry whose scales nest deeper than a walk's stack: it is compiled here by itself and its trees are
checked node by node; on the GPU hits are compared with the brute-force oracle."""
import pathlib
import shutil
import subprocess

import numpy as np
import pytest

import oracle

CSRC = next(pathlib.Path(__file__).resolve().parent.parent.glob("practical-stylized*")) / "csrc"
CHECK = r"""
#include <cstdio>
#include <functional>
#include "bvh.cuh"
using namespace sty;
using namespace sty::bvh;
int main(int, char **v) {
    FILE *f = fopen(v[1], "rb");
    std::vector<float> pos;
    float b9[9];
    while (fread(b9, 4, 9, f) == 9) pos.insert(pos.end(), b9, b9 + 9);
    const uint32_t n = (uint32_t)(pos.size() / 9);
    Builder b;
    b.pos = pos.data();
    b.build(n);
    int stack4 = 0, stack = 0, width = 0, deep = 0, most = 0, bad = 0;
    widen(b.nodes, 4, &stack4);
    const std::vector<BvhNode> w = build_wide(b.nodes, &stack, &width);
    std::function<int(uint32_t, int)> depth = [&](uint32_t i, int d) -> int {
        return b.nodes[i].count ? d : std::max(depth(b.nodes[i].a, d + 1), depth(b.nodes[i].a + 1, d + 1));
    };
    deep = depth(0, 0);
    std::vector<int> seen(n, 0);
    struct Item { uint32_t node; int held; };
    std::vector<Item> todo{{0, 0}};
    while (!todo.empty()) {
        const Item it = todo.back();
        todo.pop_back();
        const BvhNode &q = w[it.node];
        const int nc = (int)(q.exp >> 24), held = it.held + nc - 1;  // on the stack while the last child is walked
        most = std::max(most, held);
        for (int c = 0; c < nc; c++) {
            const uint32_t cnt = (q.count >> (8 * c)) & 255u;
            if (!cnt) {
                todo.push_back({q.child[c], held});
                continue;
            }
            if (cnt > 4) bad++;
            for (uint32_t k = q.child[c]; k < q.child[c] + cnt; k++) {
                seen[b.idx[k]]++;
                for (int a = 0; a < 3; a++) {  // the child's box holds its triangles
                    const double step = std::ldexp(1.0, (int)((q.exp >> (8 * a)) & 255u) - 127), o = q.o[a];
                    const double lo = o + ((q.lo[a] >> (8 * c)) & 255u) * step, hi = o + ((q.hi[a] >> (8 * c)) & 255u) * step;
                    const Box &t = b.tbox[b.idx[k]];
                    const bool all = ((q.exp >> (8 * a)) & 255u) == 254u && q.hi[a] == 0xffffffffu;  // excludes nothing
                    if (!all && !(std::isfinite(o) && lo <= t.mn[a] && hi >= t.mx[a])) bad++;
                }
            }
        }
    }
    for (int s : seen) bad += s != 1;
    printf("%d %d %d %d %d %d\n", stack4, width, stack, most, deep, bad);
}
"""


def _nested(ratio, first, last):
    """Five triangles along +-x, +-y, +z at every scale from `first` down to `last`."""
    out, s = [], first
    dirs = np.array([[1, 0, 0], [-1, 0, 0], [0, 1, 0], [0, -1, 0], [0, 0, 1.0]])
    while s >= last:
        for d in dirs:
            u = np.roll(d, 1) * 0.3
            v = np.roll(d, 2) * 0.3
            out.append([(d - u - v) * s, (d + 2 * u - v) * s, (d - u + 2 * v) * s])
        s *= ratio
    return np.array(out).reshape(-1, 9).astype(np.float32)


def _soup():
    rng = np.random.default_rng(0)
    return (rng.uniform(-1, 1, (3000, 1, 3)) + rng.normal(scale=0.05, size=(3000, 3, 3))).astype(np.float32).reshape(-1, 9)


def _far(value):
    pos = _soup()[:200].copy()
    pos[7, 3] = value  # one vertex at the end of FP32's range
    return pos


# geometry -> the width its tree is given (0: any)
CASES = {
    "soup": (_soup, 4),
    "one": (lambda: _soup()[:1], 4),
    "five the same": (lambda: np.repeat(_soup()[:1], 5, 0), 4),
    "halves": (lambda: _nested(0.5, 2.0 ** 100, 2.0 ** -119), 2),
    "halves, fewer": (lambda: _nested(0.5, 2.0 ** 50, 2.0 ** -30), 3),
    "far": (lambda: _far(3.4e38), 0),
    "far below": (lambda: _far(-3.4e38), 0),
    "tenths off": (lambda: _nested(0.9, 1e30, 1e-36), 0),
    "a twentieth off": (lambda: _nested(0.95, 1e37, 1e-37), 0),
}


def _tree(tmp_path, pos):
    gxx = shutil.which("g++")
    if not gxx:
        pytest.skip("g++ not available")
    src, exe, data = tmp_path / "check.cpp", tmp_path / "check", tmp_path / "pos.bin"
    src.write_text(CHECK)
    data.write_bytes(np.ascontiguousarray(pos, np.float32).tobytes())
    subprocess.run([gxx, "-std=c++17", "-O1", "-x", "c++", "-I", str(CSRC), str(src), "-o", str(exe)], check=True)
    return [int(v) for v in subprocess.run([str(exe), str(data)], check=True, capture_output=True, text=True).stdout.split()]


@pytest.mark.parametrize("name", CASES)
def test_tree(tmp_path, name):
    make, want = CASES[name]
    stack4, width, stack, most, deep, bad = _tree(tmp_path, make())
    assert bad == 0  # every triangle in one leaf, inside its box
    assert most == stack and stack <= 96 and deep <= 96
    assert want in (0, width) and (width == 4) == (stack4 <= 96)


@pytest.mark.gpu
@pytest.mark.parametrize("name", ["halves", "halves, fewer", "tenths off"])
def test_hits(sty, cuda, name):
    """Rays at the triangles of scales 2^-30 to 2^40, whose own products neither overflow nor underflow, from beside them."""
    import torch
    pos = CASES[name][0]()
    size = np.abs(pos).max(1)
    mid = np.flatnonzero((size > 2.0 ** -30) & (size < 2.0 ** 40))
    rng = np.random.default_rng(1)
    pick = rng.choice(mid, 3000)
    tri = pos[pick].reshape(-1, 3, 3).astype(np.float64)
    b = rng.dirichlet([1, 1, 1], pick.size)
    p = (b[:, :, None] * tri).sum(1)
    s = np.linalg.norm(p, axis=1, keepdims=True)
    o = p * 0.9 + s * rng.uniform(0.3, 0.6, (pick.size, 3)) * np.sign(rng.normal(size=(pick.size, 3)))
    d = (p - o) / np.linalg.norm(p - o, axis=1, keepdims=True)
    rays = np.concatenate([o, d, np.zeros((pick.size, 1)), 2 * np.linalg.norm(p - o, axis=1, keepdims=True)], 1).astype(np.float32)
    _, _, mats, cam = sty.scene.cornell_box(8, 8)
    sc = sty.scene.Scene(pos, np.zeros(len(pos), np.uint32), mats, cam)
    prim, t, bary = sc.closest_hit(torch.from_numpy(rays).cuda())
    rp, rt, rb = oracle.closest_hit(pos, rays)
    hit = rp != 0xFFFFFFFF
    assert hit.mean() > 0.8
    assert (prim.cpu().numpy().view(np.uint32) == rp).all()
    assert (t.cpu().numpy()[hit] == rt[hit]).all() and (bary.cpu().numpy()[hit] == rb[hit]).all()
    sc.close()


@pytest.mark.gpu
@pytest.mark.parametrize("value", [3.4e38, -3.4e38, 1e30])
def test_hits_beside_a_far_vertex(sty, cuda, value):
    """A triangle that reaches to the end of the range hides none of the others."""
    import torch
    pos = _far(value)
    rng = np.random.default_rng(3)
    aim = pos[rng.integers(8, len(pos), 3000)].reshape(-1, 3, 3).mean(1)
    o = aim + rng.normal(size=(3000, 3))
    d = (aim - o) / np.linalg.norm(aim - o, axis=1, keepdims=True)
    rays = np.concatenate([o, d, np.zeros((3000, 1)), np.full((3000, 1), 1e20)], 1).astype(np.float32)
    _, _, mats, cam = sty.scene.cornell_box(8, 8)
    sc = sty.scene.Scene(pos, np.zeros(len(pos), np.uint32), mats, cam)
    prim, t, bary = sc.closest_hit(torch.from_numpy(rays).cuda())
    rp, rt, rb = oracle.closest_hit(pos, rays)
    assert (rp != 0xFFFFFFFF).mean() > 0.9
    assert (prim.cpu().numpy().view(np.uint32) == rp).all()
    sc.close()
