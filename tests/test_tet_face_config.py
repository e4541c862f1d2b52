"""The index of a tetrahedron face in the table of face mass matrices (CPU):
inside the table for whatever local vertices a face table names, and one
place for each way a face can sit in its two elements."""
import ctypes
import itertools
import os
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
SRC = os.path.join(HERE, "hostcheck", "tet_face_host.cu")


@pytest.fixture(scope="module")
def config(tmp_path_factory):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(nvcc):
        pytest.skip("nvcc not available")
    lib = str(tmp_path_factory.mktemp("hostcheck") / "libtet_face_host.so")
    subprocess.check_call([nvcc, "-O2", "-std=c++17", "-Xcompiler", "-fPIC", "-shared", "-o", lib, SRC])
    f = ctypes.CDLL(lib).host_tet_face_config
    return lambda lo, ln: f(bytes(lo), bytes(ln))


def test_every_triple_stays_in_the_table(config):
    """A face table may name a vertex twice (its area is zero): all 64 x 64
    pairs of triples, distinct or not."""
    for lo in itertools.product(range(4), repeat=3):
        for ln in itertools.product(range(4), repeat=3):
            assert 0 <= config(lo, ln) < 96, (lo, ln)


def test_one_place_for_each_way_a_face_can_sit(config):
    """96 places: the owner's side, and the neighbour's vertex at each of the
    owner's three in ascending order; the face's own order does not matter."""
    places = {}
    for lo in itertools.permutations(range(4), 3):
        for ln in itertools.permutations(range(4), 3):
            way = (tuple(sorted(lo)), tuple(n for _, n in sorted(zip(lo, ln))))
            places.setdefault(way, set()).add(config(lo, ln))
    assert len(places) == 96 and all(len(v) == 1 for v in places.values())
    assert set().union(*places.values()) == set(range(96))
