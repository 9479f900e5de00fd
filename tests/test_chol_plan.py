"""The host-side plan of the tiled sparse Cholesky (order, fill, products,
assembly lists, order of the tiles) against its definition, without a GPU."""

import os
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "..", "g2o_b200", "csrc")


@pytest.fixture(scope="module")
def plan(tmp_path_factory):
    exe = str(tmp_path_factory.mktemp("plan") / "chol_plan_check")
    subprocess.run(["g++", "-std=c++17", "-O2", "-I", CSRC, "-o", exe, os.path.join(HERE, "chol_plan_check.cpp"),
                    os.path.join(CSRC, "chol_plan.cpp")], check=True)

    def run(kind, nb, bs, reorder=True, status=0):
        r = subprocess.run([exe, kind, str(nb), str(bs), str(int(reorder))], capture_output=True, text=True,
                           timeout=300)
        if status:
            assert r.returncode == status, (r.returncode, r.stderr)
            return None
        assert r.returncode == 0, (r.returncode, r.stdout, r.stderr)
        return [int(v) for v in r.stdout.split()]

    return run


@pytest.mark.parametrize("kind", ["chain", "star", "hubchain", "hubs", "starloops", "random", "grid", "full"])
@pytest.mark.parametrize("nb,bs", [(1, 3), (21, 3), (22, 3), (43, 6), (300, 3), (260, 6), (150, 9)])
@pytest.mark.parametrize("reorder", [True, False])
def test_plan_is_what_it_is_defined_to_be(plan, kind, nb, bs, reorder):
    if kind == "full" and nb == 260:
        nb = 160
    plan(kind, nb, bs, reorder)


# a vertex next to all others does not make the rest of the graph dense: the
# tiles and products grow with the graph's size, as those of a band do
@pytest.mark.parametrize("kind,nb,bs", [("star", 1000, 3), ("star", 8000, 3), ("star", 3000, 6), ("hubchain", 8000, 3),
                                        ("hubs", 8000, 3), ("starloops", 8000, 3)])
def test_hub_leaves_a_sparse_graph(plan, kind, nb, bs):
    nt, slots, products, chain = plan(kind, nb, bs)
    n = nb * bs
    assert slots <= 20 * n // 64 and products <= 100 * n // 64 and chain <= n // 64 // 3


# 2,345 dense tile columns have 2^31 products
@pytest.mark.parametrize("reorder", [False, True])
def test_plan_with_too_many_products_is_refused(plan, reorder):
    plan("full", 2345, 64, reorder, status=3)
