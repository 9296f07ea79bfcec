"""Workspace of a cyclic solve (cyclic_carve, shared by the host's allocation and the device's layout): the two forms
of CG share their vectors, so a solve takes no more than the form with the direction does (residual and direction
interleaved, F F^T p), apart from columns beyond the rows, and the arrays do not overlap."""
import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
SRC = r"""
#include <cstdio>
#include <cstdlib>
#include "%s/krans_b200/csrc/kr_types.cuh"
using namespace kr;
int main(int, char **a) {
  CyclicPlan p{};
  p.m = atoll(a[1]); p.n = atoll(a[2]); p.k_target = 4; p.ncv = 48;
  p.ldm = kr_round_up(p.m, 32); p.ldn = kr_round_up(p.n, 32); p.ldb = p.ldn; p.cap = 26;
  p.ksz = 8; p.precond = atoi(a[3]); p.grid_blocks = 1;
  const size_t bytes = cyclic_carve(p, nullptr, nullptr);
  char *b = (char *)(size_t)4096;
  CyclicDesc d{};
  cyclic_carve(p, b, &d);
  auto at = [&](const void *x) { return (long long)((const char *)x - b); };
  printf("%%zu %%lld %%lld %%lld %%lld %%lld %%lld %%lld\n", bytes, at(d.wm), at(d.cgr), at(d.cgts), at(d.cgus), at(d.rp), at(d.Ap),
         at(d.alpha));
}
""" % ROOT


@pytest.fixture(scope="module")
def carve(tmp_path_factory):
    d = tmp_path_factory.mktemp("ws")
    src, exe = d / "ws.cpp", d / "ws"
    src.write_text(SRC)
    subprocess.run(["g++", "-std=c++17", "-I/usr/local/cuda/include", str(src), "-o", str(exe)], check=True, timeout=300)
    return lambda *a: [int(x) for x in subprocess.run([str(exe), *map(str, a)], check=True, capture_output=True,
                                                      text=True).stdout.split()]


@pytest.mark.parametrize("precond", [0, 1])
@pytest.mark.parametrize("m,n", [(1, 1), (997, 1000), (30000, 10000), (1000, 30000), (4000, 4001)])
def test_cg_vectors_share_their_room(carve, m, n, precond):
    ldm, ldn = (m + 31) // 32 * 32, (n + 31) // 32 * 32
    bytes_, wm, cgr, cgts, cgus, rp, Ap, alpha = carve(m, n, precond)
    room = 8 * max(3 * ldm, ldm + 2 * ldn)
    assert wm + 8 * ldm <= cgr and cgr + room <= alpha <= cgr + room + 256
    assert rp == cgr and Ap == rp + 16 * ldm and Ap + 8 * ldm <= alpha
    assert cgts == cgr + 8 * ldm and cgus == cgts + 8 * ldn and cgus + 8 * ldn <= alpha
    # Krylov bases and work vectors, seven more, CG, preconditioner, and 100 kB of small arrays
    vectors = 8 * (27 * (ldm + ldn) + 5 * ldn + 2 * ldm) + room + (8 * 4 * ldm if precond else 0)
    assert bytes_ <= vectors + 100_000
