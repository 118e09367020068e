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


def _db(plan, M, N, K, gs, cfg=None):
    out = (ctypes.c_int * 4)()
    plan.plan_db(M, N, K, gs, SMS, None if cfg is None else (ctypes.c_int * 8)(*cfg), out)
    return tuple(out)


@pytest.mark.parametrize("gs", range(16, 1040, 16))
def test_plans_of_db_are_ones_the_kernel_takes(plan, gs):
    for M in (0, 1, 128, 129, 4096, 16384):
        for n in (1, 3, 40, 200):
            for K in (8, 264, 4096):
                bn, splits, tail_rows, tail_splits = _db(plan, M, n * gs, K, gs)
                assert bn % 16 == 0 and 16 <= bn <= 256 and gs % bn == 0
                assert 1 <= splits <= 16 and splits <= max(1, (M + 127) // 128)
                assert tail_rows == 0 or (splits == 1 and 0 < tail_rows < n * gs // bn and 2 <= tail_splits <= 16)


@pytest.mark.parametrize("M,K,N,gs,want", [
    (128, 256, 256, 256, (256, 1, 0, 1)),         # one token block
    (4096, 1024, 4096, 256, (256, 1, 0, 1)),      # 64 tiles, one wave: three splits would make three waves
    (2200, 256, 256, 128, (128, 9, 0, 1)),        # two tiles, 18 token blocks: as often as it pays
    (8192, 1024, 5120, 256, (256, 1, 2, 9)),      # 80 tiles: the last wave's rows are split, not everything
    (16384, 1024, 5120, 256, (256, 1, 2, 9)),
    (10031, 1728, 2816, 64, (64, 1, 2, 5)),       # narrow tiles: a block takes 0.97 us, not 1.3
    (61, 464, 224, 224, (32, 1, 0, 1)),           # one block and few tiles: narrow ones
    (2000, 3000, 6144, 192, (192, 1, 2, 3)),      # 384 tiles, the last of six waves 14
    (16384, 4096, 14336, 256, (256, 1, 1, 4))])  # 896 tiles
def test_plan_of_db(plan, M, K, N, gs, want):
    assert _db(plan, M, N, K, gs) == want


def test_plan_of_db_given_by_hand(plan):
    assert _db(plan, 4096, 4096, 1024, 256, [128, 3, 0, 0, 0, 0, 0, 0]) == (128, 3, 0, 1)
    assert _db(plan, 8192, 5120, 1024, 256, [0, -1, 0, 0, 0, 0, 0, 0]) == (256, 1, 0, 1)
    assert _db(plan, 0, 4096, 1024, 256, [0, 4, 0, 0, 0, 0, 0, 0])[1] == 4


@pytest.mark.parametrize("bn,blocks,bf16_silu,tma", [(256, 1, 1, 1), (256, 32, 1, 1), (256, 64, 1, 0), (64, 2, 1, 1), (64, 8, 1, 0),
                                                     (16, 1, 1, 0), (256, 128, 0, 1), (32, 64, 0, 1), (16, 1, 0, 0),
                                                     (256, 1 << 24, 1, 0)])
def test_which_tiles_of_db_leave_by_tma(plan, bn, blocks, bf16_silu, tma):
    assert plan.plan_db_tma(bn, blocks, bf16_silu) == tma


@pytest.mark.parametrize("M,K,G,gs,pairs,per", [
    (100, 64, 4, 64, 1, 1),          # four short steps in a row against four pairs side by side
    (100, 64, 1, 64, 1, 1),          # nothing to split
    (1024, 768, 3, 256, 24, 3),      # the sums of dA cost what two of three steps save
    (1024, 4096, 60, 64, 37, 30),    # room for two parts
    (1024, 4096, 60, 64, 38, 60),    # more than half of the pairs in use
    (128, 4096, 56, 256, 32, 28)])
def test_group_parts_of_dadr(plan, M, K, G, gs, pairs, per):
    assert plan.plan_dadr_per_part(M, K, G, gs, pairs, SMS // 2) == per


def test_group_parts_of_dadr_fit_the_pairs(plan):
    for G in (1, 2, 3, 7, 56, 1000):
        for pairs in (1, 2, 30, 37, 38, 74, 200):
            for gs in (16, 256, 1024):
                per = plan.plan_dadr_per_part(300, 1000, G, gs, pairs, SMS // 2)
                parts = -(-G // per)
                assert 1 <= per <= G and (parts == 1 or parts * pairs <= SMS // 2)
