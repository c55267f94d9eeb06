"""The device BVH build's kernels run on the CPU under the address sanitizer:
pieces whose boxes overflow float (an infinite side times a flat one is no
number) stay in bounds and are refused as too large, and ordinary pieces keep
every triangle."""

import numpy as np
import pytest

from tests import device_host

PROGRAM = r"""
#include <algorithm>
#include <cstdio>
#include <numeric>
#include "argent_b200/csrc/device_build.cuh"
using host_emulation::launch;
// Input: nv, nt, positions, indices.  Output: err, node count, triangles, and
// the original triangle of each record.
int main() {
  uint32_t nv, nt;
  if (fread(&nv, 4, 1, stdin) != 1 || fread(&nt, 4, 1, stdin) != 1) return 1;
  std::vector<float> pos(3 * nv);
  std::vector<uint32_t> tri(3 * nt);
  if (fread(pos.data(), 12, nv, stdin) != nv || fread(tri.data(), 12, nt, stdin) != nt) return 1;
  const size_t nb = 2 * (size_t)nt - 1;
  std::vector<float4> pos4(nv), tris(3 * (size_t)nt);
  std::vector<uint4> tidx(nt), nodes(5 * (size_t)std::max(1u, nt - 1));
  std::vector<uint32_t> info(8), vals(nt), first(nb), last(nb), flag(nb), ctr(68);
  std::vector<float> tlo(3 * nt), thi(3 * nt), cen(3 * nt), lo(3 * nb), hi(3 * nb);
  std::vector<uint64_t> keys(nt), sorted(nt);
  std::vector<int32_t> left(nb), right(nb), parent(nb);
  launch(1, 256, [&] {
    db::k_piece_pack(pos.data(), nullptr, tri.data(), nullptr, nv, nt, pos4.data(), nullptr, tidx.data(), info.data());
  });
  if (info[0]) return 2;
  launch(1, 256, [&] { db::k_tri_boxes(pos4.data(), tidx.data(), nt, tlo.data(), thi.data(), cen.data(), info.data() + 2); });
  launch(1, 32, [&] { db::k_morton(cen.data(), nt, info.data() + 2, keys.data(), vals.data()); });
  std::vector<uint32_t> order(nt);
  std::iota(order.begin(), order.end(), 0u);
  std::stable_sort(order.begin(), order.end(), [&](uint32_t a, uint32_t b) { return keys[a] < keys[b]; });
  for (uint32_t i = 0; i < nt; ++i) sorted[i] = keys[order[i]];
  vals = order;
  db::Bin bn{lo.data(), hi.data(), first.data(), last.data(), left.data(), right.data(), parent.data(), flag.data()};
  launch(1, 32, [&] { db::k_radix_tree(sorted.data(), nt, bn); });
  launch(1, 32, [&] { db::k_boxes_up(tlo.data(), thi.data(), vals.data(), nt, bn); });
  std::vector<int2> qa(nt), qb(nt);
  qa[0] = make_int2(0, 0);
  ctr[0] = 1;
  ctr[65] = 1;
  db::Collapse c{};
  c.node_count = ctr.data() + 65;
  c.tri_count = ctr.data() + 66;
  c.err = ctr.data() + 67;
  c.nodes = nodes.data();
  c.tris = tris.data();
  c.pos = pos4.data();
  c.tri = tidx.data();
  c.vals = vals.data();
  for (uint32_t level = 0; level < 64 && ctr[level]; ++level) {
    c.in = level & 1 ? qb.data() : qa.data();
    c.out = level & 1 ? qa.data() : qb.data();
    c.n_in = ctr.data() + level;
    c.n_out = ctr.data() + level + 1;
    launch(1, 64, [&] { db::k_collapse(c, bn, nt); });
  }
  fwrite(ctr.data() + 67, 4, 1, stdout);
  fwrite(ctr.data() + 65, 4, 2, stdout);
  for (uint32_t i = 0; i < nt; ++i) fwrite(&tris[3 * (size_t)i].w, 4, 1, stdout);
}
"""

ERR_EXTENT, ERR_QUANT = 1, 2


def _strips(n, far, rng):
    """2 n small triangles flat in y: half near x = 0 and half at x = +-far, so
    that some binary nodes span 2 far by nothing and others are ordinary."""
    c = np.zeros((2 * n, 3))
    c[:, 2] = np.arange(2 * n)
    c[n:, 0] = far * rng.choice([-1.0, 1.0], n)
    corner = np.array([[0, 0, 0], [0.5, 0, 0], [0, 0, 0.5]])
    pos = (c[:, None] + corner).reshape(-1, 3).astype(np.float32)
    return pos, np.arange(6 * n, dtype=np.uint32).reshape(-1, 3)


@pytest.fixture(scope="module")
def program(tmp_path_factory):
    return device_host.compile_program(PROGRAM, str(tmp_path_factory.mktemp("build")), sanitize=True)


@pytest.mark.parametrize("far", [5.0, 1e30, 3e38])
@pytest.mark.parametrize("n", [3, 16, 70])
def test_collapse_stays_in_bounds(program, n, far):
    pos, tris = _strips(n, far, np.random.default_rng(n))
    data = np.uint32([len(pos), len(tris)]).tobytes() + pos.tobytes() + tris.tobytes()
    out = np.frombuffer(device_host.run(program, data), np.uint32)
    err, nodes, count, prims = out[0], out[1], out[2], out[3:]
    assert (err != 0) == (far > 1e20)
    assert 0 < nodes < len(tris) and count == len(tris)
    assert np.array_equal(np.sort(prims), np.arange(len(tris)))


@pytest.mark.gpu
def test_boxes_that_overflow_are_refused():
    from argent_b200 import mesh as M
    from argent_b200._native import ArgentError
    from argent_b200.gpu import Context, Piece

    ctx = Context(0)
    for n in (3, 16, 70):
        pos, tris = _strips(n, 3e38, np.random.default_rng(n))
        with pytest.raises(ArgentError):
            Piece(ctx, M.Mesh(pos, tris), device_bvh=True)
    pos, tris = _strips(70, 5.0, np.random.default_rng(70))
    piece = Piece(ctx, M.Mesh(pos, tris), device_bvh=True)
    rays = np.zeros((len(tris), 8), np.float32)
    rays[:, :3] = pos[::3] + np.float32([0.1, 1.0, 0.1])
    rays[:, 3], rays[:, 5] = np.inf, -1.0
    assert np.array_equal(piece.trace_closest(rays)[:, 3].view(np.uint32), np.arange(len(tris)))
