"""The two-step division and the packed masses of csrc/common.cuh against CUDA's own division and the scalar form, over whole ranges
of operands (tests/mass_probe.cu, compiled here)."""
import ctypes as C
import os
import subprocess

import pytest
import torch

from colinfer_b200 import build

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def probe(tmp_path_factory):
    so = str(tmp_path_factory.mktemp("probe") / "mass_probe.so")
    src = os.path.join(os.path.dirname(os.path.abspath(__file__)), "mass_probe.cu")
    subprocess.run([os.environ.get("NVCC", "nvcc"), *build.NVCC_FLAGS, "-shared", src, "-o", so], check=True, capture_output=True)
    lib = C.CDLL(so)
    lib.probe_quotients.argtypes = [C.c_void_p, C.c_int, C.c_int, C.c_void_p]
    lib.probe_masses.argtypes = [C.c_void_p, C.c_void_p, C.c_int, C.c_void_p]
    return lib


def _temperatures():
    g = torch.Generator().manual_seed(7)
    t = torch.cat([torch.tensor([1e-6, 0.01, 0.3, 0.5, 0.7, 0.8, 0.9, 1.0, 1.1, 1.5, 2.0, 100.0]), 0.05 + 2.0 * torch.rand(52, generator=g)])
    return t.float().cuda()


@pytest.mark.parametrize("exp0", [-60, -20, -1, 0, 3, 60])
def test_the_two_step_quotient_is_the_ieee_one(probe, exp0):
    t = _temperatures()
    bad = torch.zeros(len(t), 2, dtype=torch.int64, device="cuda")
    assert probe.probe_quotients(t.data_ptr(), len(t), exp0, bad.data_ptr()) == 0
    assert int(bad.sum()) == 0, (t[bad[:, 0] > 0].tolist(), bad[bad[:, 0] > 0].tolist())


def test_a_significand_of_all_ones_leaves_it_a_unit_off_at_most(probe):
    t = (torch.tensor([0x3FFFFFFF, 0x3F7FFFFF, 0x3EFFFFFF, 0x42FFFFFF], dtype=torch.int32).view(torch.float32)).cuda()
    for exp0 in (-3, 0, 4):
        bad = torch.zeros(len(t), 2, dtype=torch.int64, device="cuda")
        assert probe.probe_quotients(t.data_ptr(), len(t), exp0, bad.data_ptr()) == 0
        assert int(bad[:, 1].sum()) == 0


def test_packed_masses_are_the_scalar_ones(probe):
    t = _temperatures()
    lmax = 30.0 * torch.rand(len(t), generator=torch.Generator().manual_seed(8)).cuda() - 5.0
    bad = torch.zeros(len(t), dtype=torch.int64, device="cuda")
    assert probe.probe_masses(t.data_ptr(), lmax.data_ptr(), len(t), bad.data_ptr()) == 0
    assert int(bad.sum()) == 0
