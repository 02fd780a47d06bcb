"""A wait of a moment loop that runs out is reported wherever a set reaches the host. The
kernels flag it in the Hamiltonian's device word; here a small C++ helper sets that word from
the host, as the kernel would, and no wait runs out."""
from __future__ import annotations

import ctypes
import os
import subprocess

import numpy as np
import pytest

import gpuqt_b200 as g
from conftest import ROOT, fixture_dir

pytestmark = pytest.mark.gpu

HELPER = r"""
#include <cstdio>
#include <cstdlib>
#include "gqt_internal.h"
#include "lsqt/hamiltonian.h"
#include "lsqt/model.h"
#include "lsqt/sigma.h"
#include "lsqt/vector.h"
extern "C" int set_flag(gqt_ham* h, unsigned bits)
{
  return cudaMemcpy(h->stage_err, &bits, sizeof(bits), cudaMemcpyHostToDevice);
}
int main(int, char** argv)
{
  Model model(argv[1]);
  Hamiltonian H(model);
  Vector phi(model.number_of_atoms), mu(model.number_of_moments);
  model.initialize_state(phi, -1);
  if (set_flag(H.handle(), (unsigned)atoi(argv[2])))
    return 9;
  find_moments_chebyshev(model, H, phi, phi, mu);
  puts("returned");
  return 0;
}
"""
LOOPS = {1: "staged step", 2: "strip loop"}


def _compile(tmp, shared):
    src, out = os.path.join(tmp, "h.cpp"), os.path.join(tmp, "h.so" if shared else "h")
    with open(src, "w") as f:
        f.write(HELPER)
    lib = os.path.dirname(g.LIB_PATH)
    cuda = os.environ.get("CUDA_HOME", "/usr/local/cuda")
    subprocess.run(["g++", "-std=c++17", *(["-shared", "-fPIC"] if shared else []), src, "-o", out,
                    f"-I{ROOT}/include", f"-I{ROOT}/gpuqt_b200/csrc", f"-I{cuda}/include",
                    f"-L{lib}", "-lgpuqt_b200", f"-Wl,-rpath,{lib}", f"-L{cuda}/lib64",
                    "-lcudart_static", "-lpthread", "-ldl", "-lrt"], check=True)
    return out


@pytest.mark.parametrize("bits", sorted(LOOPS))
def test_flag_is_reported_once_by_each_entry(bits, tmp_path):
    import torch

    helper = ctypes.CDLL(_compile(str(tmp_path), True))
    m = g.Model.load(fixture_dir("sq16_pbc"))
    H = g.Hamiltonian(m)
    x = g.Vector.from_host(*m.initial_state())
    M = 20
    want = g.moments(H, x, x, M)
    mu = torch.zeros(M, dtype=torch.complex128, device="cuda")

    def flagged(call):
        assert helper.set_flag(H.h, ctypes.c_uint(bits)) == 0
        with pytest.raises(g.GqtError, match=LOOPS[bits]):
            call()
        g.check_moments(H)  # reported once
        got = g.moments(H, x, x, M)
        assert np.array_equal(got[0], want[0]) and np.array_equal(got[1], want[1])

    flagged(lambda: g.moments(H, x, x, M))
    flagged(lambda: g.moments_doubled(H, x, M))

    def device():
        torch.cuda.synchronize()
        g.moments_device(H, x, x, M, mu.data_ptr())
        g.check_moments(H)

    flagged(device)
    assert np.array_equal(mu.cpu().numpy(), want[0] + 1j * want[1])


def test_flag_ends_the_cxx_drivers_moments(tmp_path):
    exe = _compile(str(tmp_path), False)
    args = [exe, fixture_dir("sq16_pbc")]
    ok = subprocess.run([*args, "0"], capture_output=True, text=True)
    assert ok.returncode == 0 and "returned" in ok.stdout, ok.stderr
    bad = subprocess.run([*args, "2"], capture_output=True, text=True)
    text = bad.stdout + bad.stderr
    assert bad.returncode not in (0, 9) and "returned" not in text and "strip loop" in text
