"""The union-find operations of csrc/uf.cuh in every order, on the CPU: a
carried round of an eps sweep hooks newly core points and then unites the new
edges alone, so no order may lose a link that an earlier eps made."""
import os
import re
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(os.path.dirname(HERE), "sdbscan_gb300", "csrc")


@pytest.fixture(scope="module")
def program(tmp_path_factory):
    out = tmp_path_factory.mktemp("uf")
    with open(os.path.join(CSRC, "uf.cuh")) as f:
        src = re.sub(r"^#(pragma once|include).*$", "", f.read(), flags=re.M)
    (out / "uf_host.h").write_text(src)
    with open(os.path.join(CSRC, "common.cuh")) as f:
        limit = int(re.search(r"kCompressRounds = (\d+)", f.read()).group(1))
    exe = out / "uf_orders"
    subprocess.run(["g++", "-O2", "-std=c++17", "-w", "-U_FORTIFY_SOURCE", f"-DKCOMPRESS={limit}", f"-I{out}",
                    os.path.join(HERE, "uf_orders.cpp"), "-o", str(exe)], check=True)
    return exe, limit


def _run(exe, n, carried):
    return subprocess.run([str(exe), str(n), str(int(carried))], capture_output=True, text=True, timeout=120)


@pytest.mark.parametrize("compressed", [False, True])
def test_carried_round_keeps_the_links_of_an_earlier_eps(program, compressed):
    exe, limit = program
    r = _run(exe, limit if compressed else 6, True)
    assert r.returncode == 0, r.stdout
    assert re.match(r"540 cases, \d+ outcomes", r.stdout)


def test_the_orders_include_one_that_loses_a_link_beside_halved_paths(program):
    """The walk of the other rounds, whose union pass visits every edge."""
    exe, _ = program
    r = _run(exe, 6, False)
    assert r.returncode == 1 and r.stdout.startswith("split:")


def test_compression_leaves_every_point_at_its_root(program):
    """Labels, borders and flood starts are read from the parents after it."""
    exe, _ = program
    r = subprocess.run([str(exe), "compress"], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stdout
    assert re.match(r"\d+ cases", r.stdout)
