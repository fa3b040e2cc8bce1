"""The per-thread search (enum_core.cuh) compiled for the host with bounds checks:
every k that the library takes, up to 15, stays inside its arrays and finds the
oracle's set."""
import json
import os
import shutil
import subprocess

import pytest

import oracle as O
from gmkbe_b200 import graphgen as gg
from conftest import ROOT


@pytest.fixture(scope="module")
def search(tmp_path_factory):
    if shutil.which("g++") is None:
        pytest.skip("g++ not available")
    exe = str(tmp_path_factory.mktemp("ws") / "search")
    built = subprocess.run(["g++", "-O1", "-g", "-std=c++17", "-fsanitize=address,undefined",
                            "-fno-sanitize-recover=all", "-o", exe, os.path.join(ROOT, "oracle", "work_count.cpp")],
                           capture_output=True, text=True)
    if built.returncode:
        pytest.skip("no address sanitizer: " + built.stderr[-200:])
    return exe


@pytest.mark.parametrize("nu,nv,p,k", [(6, 14, 0.5, 4), (7, 9, 0.6, 3), (9, 8, 0.8, 4), (8, 9, 0.85, 5),
                                       (9, 9, 0.9, 6), (10, 10, 0.95, 7), (11, 11, 1.0, 8),
                                       (10, 30, 0.04, 15)])
def test_every_k_within_its_arrays(search, tmp_path, nu, nv, p, k):
    g = gg.erdos_renyi(nu, nv, p, 3)
    path = str(tmp_path / "g.graph.bin")
    gg.write_graph_bin(g, path)
    out = subprocess.run([search, path, str(k)], capture_output=True, text=True, timeout=120)
    assert out.returncode == 0, out.stderr[:1500]
    r = json.loads(out.stdout)
    assert (r["results"], int(r["hash_sum"], 16), int(r["hash_xor"], 16)) == O.enumerate_oracle(g, k).summary()
