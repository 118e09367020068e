"""The rules that choose tile widths and splits from sizes, called on the CPU (148 SMs, 74 CTA pairs)."""
import ctypes
import os
import subprocess

import pytest

SMS = 148


@pytest.fixture(scope="module")
def plan(tmp_path_factory):
    here = os.path.dirname(os.path.abspath(__file__))
    so = str(tmp_path_factory.mktemp("plan") / "libplan_probe.so")
    subprocess.run(["g++", "-std=c++17", "-Wall", "-Werror", "-shared", "-fPIC", "-o", so,
                    os.path.join(here, "csrc", "plan_probe.cpp")], check=True)
    L = ctypes.CDLL(so)
    L.plan_fwd_us.restype = ctypes.c_double
    return L


@pytest.mark.parametrize("gs", range(16, 1040, 16))
@pytest.mark.parametrize("bias", [0, 1])
def test_forward_tile_widths_are_ones_the_kernel_takes(plan, gs, bias):
    for M in (1, 256, 257, 4096, 16384):
        for n in (1, 3, 40):
            for K in (8, 4096):
                bn = plan.plan_fwd_bn(M, n * gs, K, gs, bias, SMS)
                assert bn % 16 == 0 and 16 <= bn <= 256 and gs % bn == 0


@pytest.mark.parametrize("M,K,N,gs,bias,bn", [
    (300, 1024, 768, 192, 1, 64), (300, 1024, 768, 192, 0, 64),     # a wave of narrow tiles with TMA stores, not 96 wide
    (207, 496, 448, 224, 1, 32), (207, 496, 448, 224, 0, 32),       # plain stores cost more the wider the tile
    (165, 120, 1568, 224, 1, 32),
    (1000, 1000, 1440, 96, 0, 96), (2000, 3000, 6144, 192, 1, 192), # enough tiles: the widest
    (4096, 1024, 4480, 224, 1, 224),
    # powers of two: halved while one wave holds them
    (1, 4096, 256, 256, 0, 64), (1024, 256, 1024, 256, 1, 64), (257, 768, 1024, 256, 0, 64), (128, 4096, 14336, 256, 0, 256),
    (256, 512, 18944, 256, 0, 256), (300, 512, 4608, 512, 1, 128), (64, 512, 512, 32, 1, 32), (64, 512, 528, 48, 1, 16)])
def test_forward_tile_width(plan, M, K, N, gs, bias, bn):
    assert plan.plan_fwd_bn(M, N, K, gs, bias, SMS) == bn
