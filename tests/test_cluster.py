"""The single-body PCG inside one thread-block cluster (kPcgCluster): its host
partition (tl_cluster_build.h, compiled with g++), and on the GPU its solves
against the element-by-element form, at the sizes where the partition changes:
fewer slices than blocks, whole and broken slices, 4 and 8 slices a block (the
workers that share a slice, the owners of one slice), the largest body and one
past it."""
import os
import shutil
import subprocess

import numpy as np
import pytest

import talus_b200 as tb
from tests.helpers import DT, GRAVITY, relative_error
from tests.test_sell_build import CSRC, incidence

DRIVER = r"""
#include "tl_cluster_build.h"
#include <cstdio>
using namespace tl;
int main(int argc, char** argv) {
  FILE* f = std::fopen(argv[1], "rb");
  uint32_t n[4];
  if (std::fread(n, 4, 4, f) != 4) return 2;
  const uint32_t rows = n[0], T = n[1], E = n[2], ctas = n[3];
  std::vector<uint32_t> tets(4 * size_t(T)), start(size_t(rows) + 1), entry(E);
  if (std::fread(tets.data(), 4, tets.size(), f) != tets.size()) return 2;
  if (std::fread(start.data(), 4, start.size(), f) != start.size()) return 2;
  if (std::fread(entry.data(), 4, entry.size(), f) != entry.size()) return 2;
  std::fclose(f);
  const SellHost h = buildSellHost(rows, tets.data(), start, entry);
  ClusterHost c;
  if (!buildClusterHost(h, ctas, c)) return 3;
  // each block's vector as the kernel fills it: its own rows, then what the rows' owners send
  std::vector<std::vector<int64_t>> vec(ctas);
  std::vector<uint32_t> got(ctas, 0);
  const auto put = [&](uint32_t code, uint32_t row) {
    std::vector<int64_t>& v = vec[code >> 16];
    if ((code & 0xffffu) >= v.size() || v[code & 0xffffu] >= 0) return false;
    v[code & 0xffffu] = row;
    ++got[code >> 16];
    return true;
  };
  for (uint32_t q = 0; q < ctas; ++q) {
    const uint32_t lo = clusterSlice(h.slices, ctas, q) * SELL_ROWS, hi = clusterSlice(h.slices, ctas, q + 1) * SELL_ROWS;
    vec[q].assign(hi - lo + c.foreign[q], -1);
    if (vec[q].size() > c.maxEntries) return 4;
    for (uint32_t r = lo; r < hi; ++r) vec[q][r - lo] = r;
  }
  for (uint32_t r = 0; r < h.slices * SELL_ROWS; ++r) {
    for (uint32_t d = 0; d < CLUSTER_INLINE; ++d)
      if (c.push[CLUSTER_INLINE * size_t(r) + d] != CLUSTER_NO_PUSH && !put(c.push[CLUSTER_INLINE * size_t(r) + d], r)) return 5;
    for (uint32_t o = c.overStart[r]; o < c.overStart[r + 1]; ++o)
      if (!put(c.over[o], r)) return 5;
  }
  for (uint32_t q = 0; q < ctas; ++q) {
    if (got[q] != c.foreign[q]) return 6;  // the bytes a block waits for
    const uint32_t a = clusterSlice(h.slices, ctas, q), b = clusterSlice(h.slices, ctas, q + 1);
    if (h.sliceStart[b] - h.sliceStart[a] > c.maxPositions) return 7;
    for (uint32_t p = h.sliceStart[a]; p < h.sliceStart[b]; ++p) {
      const uint32_t row = h.groupSlice[p / SELL_ROWS] * SELL_ROWS + p % SELL_ROWS;
      if (vec[q][c.local[p]] != int64_t(row < rows ? h.col[p] : row)) return 8;
    }
  }
  std::printf("%u\n", h.slices);
  return 0;
}
"""


def renumbered(mesh, seed):
    """The mesh with its nodes in random order: rows whose columns are spread over every block."""
    order = np.random.default_rng(seed).permutation(mesh.nodes)
    rank = np.argsort(order)
    return tb.PreparedMesh(mesh.rest_positions[order], mesh.node_mass[order], mesh.anchored[order],
                           rank[mesh.tet_nodes].astype(np.uint32), mesh.rest_inverse, mesh.volume, mesh.material)


@pytest.fixture(scope="module")
def driver(tmp_path_factory):
    gxx = shutil.which("g++")
    if gxx is None:
        pytest.skip("g++ not available")
    d = tmp_path_factory.mktemp("cluster")
    (d / "driver.cc").write_text(DRIVER)
    subprocess.run([gxx, "-O1", "-std=c++17", "-I", CSRC, str(d / "driver.cc"), "-o", str(d / "driver")], check=True)
    return d


@pytest.mark.parametrize("cells,shuffle", [((1, 1, 1), False), ((1, 1, 7), False), ((7, 7, 7), False),
                                           ((8, 9, 10), False), ((6, 5, 7), True)])
@pytest.mark.parametrize("ctas", [4, 16])
def test_every_column_is_in_its_blocks_vector(driver, cells, shuffle, ctas):
    mesh = tb.box_mesh(cells, voxel=0.1)
    if shuffle:
        mesh = renumbered(mesh, 1)
    start, entry = incidence(mesh.tet_nodes, mesh.nodes)
    path = os.path.join(driver, "in.bin")
    with open(path, "wb") as f:
        np.array([mesh.nodes, mesh.tets, entry.size, ctas], np.uint32).tofile(f)
        for a in (np.ascontiguousarray(mesh.tet_nodes, np.uint32), start, entry):
            a.tofile(f)
    out = subprocess.run([os.path.join(driver, "driver"), path], capture_output=True, text=True)
    assert out.returncode == 0
    assert int(out.stdout) == (mesh.nodes + 31) // 32


# (cells, renumbered): 8 nodes; one whole slice; 16 slices; 18; 64 (4 a block); 72; 128 (8 a block); 136 (two slices
# an owner); 160, the most; 170, past it
SIZES = [((1, 1, 1), False), ((1, 1, 7), False), ((7, 7, 7), False), ((8, 7, 7), False), ((7, 15, 15), False),
         ((8, 14, 16), False), ((15, 15, 15), False), ((15, 16, 15), False), ((15, 19, 15), False),
         ((15, 19, 16), False), ((6, 5, 7), True), ((15, 16, 15), True)]


@pytest.mark.gpu
@pytest.mark.parametrize("cells,shuffle", SIZES)
@pytest.mark.parametrize("precision,tol", [(tb.FP64, 1e-10), (tb.FP32_MIXED, 1e-5)])
def test_cluster_solves_match_the_elementwise_form(cells, shuffle, precision, tol):
    mesh = tb.box_mesh(cells, voxel=0.1, jitter=0.01, seed=3)
    if shuffle:
        mesh = renumbered(mesh, 2)
    mat = tb.PhysicalMaterial(density=1000.0, youngs_modulus=1e6, poissons_ratio=0.3)
    out = {}
    for form in ("auto", "elementwise"):
        s = tb.System(mesh, [mat], precision)
        s.set_solver(form)
        s.set_state(tb.rest_state(mesh))
        its = [s.step(tb.Settings(), GRAVITY, DT)[0].cg_iterations for _ in range(4)]
        out[form] = s.get_state().position, its
        s.close()
    assert relative_error(out["auto"][0], out["elementwise"][0], mesh.rest_positions) <= tol
    if precision == tb.FP64:
        assert out["auto"][1] == out["elementwise"][1]


@pytest.mark.gpu
@pytest.mark.parametrize("cells", [(1, 1, 1), (1, 1, 7), (7, 7, 7)])
@pytest.mark.parametrize("precision", [tb.FP64, tb.FP32_MIXED])
def test_blocks_of_one_owner_take_the_same_decisions(cells, precision):
    """Bodies of at most 16 slices: one warp of a block owns its rows, and its lanes each send the block's sums, which
    lane 0 wrote, to another block.  Every block has to see the same sums, so a repeated solve is bitwise the same."""
    mesh = tb.box_mesh(cells, voxel=0.1, jitter=0.01, seed=3)
    mat = tb.PhysicalMaterial(density=1000.0, youngs_modulus=1e7, poissons_ratio=0.3)
    s = tb.System(mesh, [mat], precision)
    out = []
    for _ in range(8):
        s.set_state(tb.rest_state(mesh))
        its = [s.step(tb.Settings(tolerance=1e-6, cg_iterations=500), GRAVITY, DT)[0].cg_iterations for _ in range(4)]
        out.append((its, s.get_state().position))
    s.close()
    for its, x in out[1:]:
        assert its == out[0][0]
        assert np.array_equal(x, out[0][1])


@pytest.mark.gpu
@pytest.mark.parametrize("cells", [(1, 1, 7), (8, 7, 7), (15, 16, 15)])
def test_operator_applications_are_those_of_the_elementwise_form(cells):
    """The same order and in FP64 the same iterations, so the same products with the operator."""
    mesh = tb.box_mesh(cells, voxel=0.1, jitter=0.01, seed=3)
    mat = tb.PhysicalMaterial(density=1000.0, youngs_modulus=1e6, poissons_ratio=0.3)
    out = {}
    for form in ("auto", "elementwise"):
        s = tb.System(mesh, [mat], tb.FP64)
        s.set_solver(form)
        s.set_state(tb.rest_state(mesh))
        reports = [s.step(tb.Settings(cg_iterations=1000), GRAVITY, DT)[0] for _ in range(3)]
        out[form] = [(r.cg_iterations, r.operator_applications) for r in reports]
        s.close()
    assert out["auto"] == out["elementwise"]


def scattered(mesh, share, seed):
    """The mesh with a share of its nodes renumbered among themselves."""
    order = np.arange(mesh.nodes)
    some = np.random.default_rng(seed).permutation(mesh.nodes)[:int(share * mesh.nodes)]
    order[np.sort(some)] = some
    rank = np.argsort(order)
    return tb.PreparedMesh(mesh.rest_positions[order], mesh.node_mass[order], mesh.anchored[order],
                           rank[mesh.tet_nodes].astype(np.uint32), mesh.rest_inverse, mesh.volume, mesh.material)


@pytest.mark.gpu
@pytest.mark.parametrize("cells,share,cluster", [((15, 16, 15), 0.0, True), ((15, 16, 15), 0.1, True),
                                                 ((15, 16, 15), 1.0, False), ((9, 9, 9), 1.0, True)])
@pytest.mark.parametrize("precision,tol", [(tb.FP64, 1e-10), (tb.FP32_MIXED, 1e-5)])
def test_nodes_in_no_order_of_place(cells, share, cluster, precision, tol):
    """A body whose blocks read too many foreign rows solves over the whole grid, which takes one more launch a solve;
    one with a tenth of its nodes scattered (rows that more than four blocks read) stays in the cluster."""
    mesh = scattered(tb.box_mesh(cells, voxel=0.1, jitter=0.01, seed=3), share, 2)
    mat = tb.PhysicalMaterial(density=1000.0, youngs_modulus=1e6, poissons_ratio=0.3)
    out = {}
    for form in ("auto", "assembled-two-phase", "elementwise"):
        s = tb.System(mesh, [mat], precision)
        s.set_solver(form)
        s.set_state(tb.rest_state(mesh))
        reports = [s.step(tb.Settings(), GRAVITY, DT)[0] for _ in range(2)]
        out[form] = s.get_state().position, reports[-1]
        s.close()
    launches = {f: r.kernel_launches for f, (_, r) in out.items()}
    assert (launches["auto"] < launches["assembled-two-phase"]) == cluster
    assert relative_error(out["auto"][0], out["elementwise"][0], mesh.rest_positions) <= tol
