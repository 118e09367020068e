"""Edges of the kernels' tiles, plans and copies, against the oracle in fp32 on the same 16-bit-rounded inputs.

TOL is the reference's bar for 16-bit outputs (tests/test_correctness.py:24-31), as in test_gpu_parity.py."""
import pytest
import torch

import cute_mma_b200 as cp
from oracle import prism_oracle as O

pytestmark = pytest.mark.gpu
TOL = 2e-2
DEV = "cuda"


def _inputs(M, K, N, gs, rs, dt, seed=0):
    return [t.to(dt).to(DEV).contiguous() for t in O.make_inputs(M, K, N, gs, rs, seed=seed, b_std=K ** -0.5)]


@pytest.mark.parametrize("offset", [0, 2])          # 16-byte and 4-byte aligned bias
@pytest.mark.parametrize("gs,N", [(256, 2560), (64, 192), (96, 288)])
def test_bias_in_the_forward_epilogue(gs, N, offset):
    """Several tiles per CTA pair (a bias of its own each), narrow tiles, and the plain-store epilogue (gs 96)."""
    M, K, rs, dt = 4100, 128, 16, torch.bfloat16
    A, B, R, _ = _inputs(M, K, N, gs, rs, dt, 3)
    bias = torch.randn(N + 8, device=DEV).to(dt)[offset:offset + N]
    C, _ = cp.forward(A, B, R, gs, rs, activation="silu_gate", bias=bias)
    cp.check_device_status()
    assert O.rel_err(C.float(), O.prism_forward(A.float(), B.float(), R.float(), gs, rs, "silu_gate", bias=bias.float())) < TOL


@pytest.mark.parametrize("gs", [48, 96, 160, 192, 224, 288])
@pytest.mark.parametrize("rs", [8, 64])
def test_tile_width_of_odd_groups(gs, rs):
    """Groups whose widest tile is no power of two: forward (TMA and plain stores), dB and dA+dR."""
    M, K, N, dt, act = 300, 192, 2 * gs, torch.float16, "silu_gate"
    A, B, R, dC = _inputs(M, K, N, gs, rs, dt, 5)
    C, _ = cp.forward(A, B, R, gs, rs, activation=act)
    dA, dR, dB, _ = cp.backward(dC, A, B, R, gs, rs, activation=act)
    cp.check_device_status()
    f = [t.float() for t in (A, B, R)]
    rA, rR, rB = O.prism_backward(dC.float(), *f, gs, rs, act)
    for got, ref in ((C, O.prism_forward(*f, gs, rs, act)), (dA, rA), (dR, rR), (dB, rB)):
        assert O.rel_err(got.float(), ref) < TOL


@pytest.mark.parametrize("K,rs", [(72, 8), (2056, 8), (2080, 16)])   # one warp; past one pass of a block; odd blocks of 8
def test_widened_and_halved_rotation(K, rs):
    M, N, gs, dt, act = 130, 256, 128, torch.bfloat16, "silu_gate"
    A, B, R, dC = _inputs(M, K, N, gs, rs, dt, 7)
    C, _ = cp.forward(A, B, R, gs, rs, activation=act)
    dA, dR, dB, _ = cp.backward(dC, A, B, R, gs, rs, activation=act)
    cp.check_device_status()
    f = [t.float() for t in (A, B, R)]
    rA, rR, rB = O.prism_backward(dC.float(), *f, gs, rs, act)
    for got, ref in ((C, O.prism_forward(*f, gs, rs, act)), (dA, rA), (dR, rR), (dB, rB)):
        assert O.rel_err(got.float(), ref) < TOL


@pytest.mark.parametrize("M,K,N,gs", [(128, 256, 256, 256),       # one token block: never split
                                      (129, 272, 512, 256),       # two blocks, features past the first pair
                                      (2200, 256, 256, 128),      # few tiles: split as often as it pays
                                      (4096, 1024, 4096, 256)])   # 64 tiles: one wave, not split
@pytest.mark.parametrize("out", [None, torch.float32])
def test_split_plan_of_db(M, K, N, gs, out):
    rs, dt, act = 16, torch.bfloat16, "sigmoid_gate"
    A, B, R, dC = _inputs(M, K, N, gs, rs, dt, 9)
    dB = cp.backward(dC, A, B, R, gs, rs, activation=act, dB_dtype=out)[2]
    cp.check_device_status()
    ref = O.prism_backward(dC.float(), A.float(), B.float(), R.float(), gs, rs, act)[2]
    assert dB.dtype == (out or dt) and O.rel_err(dB.float(), ref) < TOL


@pytest.mark.parametrize("G,K,rows", [(1, 64, 1), (3, 192, 33), (5, 1088, 8)])
@pytest.mark.parametrize("dt", [torch.bfloat16, torch.float32])
def test_shuffle_copies_are_the_index_operations(G, K, rows, dt):
    """The copy kernels against the index operations of the same fold on the CPU: bit for bit, adjoints included; a matrix
    that starts in the middle of a segment is taken too."""
    from cute_mma_b200 import _shuffle as S
    masks, _ = S.build_shuffle_masks(K, G * 32, 32, 16)
    masks = masks if G > 1 else masks + 0x5A3C   # a single group is the identity otherwise
    cpu, gpu = S.ShuffleFold(masks, K, 32, 16, "cpu"), S.ShuffleFold(masks, K, 32, 16, torch.device(DEV, 0))
    X, D64 = torch.randn(G * rows, K).to(dt), torch.randn(G * 64, K).to(dt)
    off = torch.empty(G * rows * K + 1, dtype=dt, device=DEV)[1:].view(G * rows, K).copy_(X)
    for Y in (X.to(DEV), off):
        assert torch.equal(gpu.fold_cols(Y, rows).cpu(), cpu.fold_cols(X, rows))
        assert torch.equal(gpu.unfold_cols(Y, rows).cpu(), cpu.unfold_cols(X, rows))
    assert torch.equal(gpu.unfold_dR(D64.to(DEV)).cpu(), cpu.unfold_dR(D64))
    R = torch.randn(G * 16, K).to(dt)
    r_gpu, r_cpu = R.to(DEV).requires_grad_(), R.clone().requires_grad_()
    out, ref = gpu.fold_R(r_gpu), cpu.fold_R(r_cpu)
    assert torch.equal(out.detach().cpu(), ref.detach())
    out.backward(D64.to(DEV))
    ref.backward(D64)
    assert torch.equal(r_gpu.grad.cpu(), r_cpu.grad)


@pytest.mark.parametrize("M,K,p", [(1, 64, 0.5), (130, 200, 0.1), (300, 1096, 2.0 ** -24), (257, 136, 0.999)])
@pytest.mark.parametrize("ib", [False, True])
def test_dropout_mask_of_the_dadr_kernel(M, K, p, ib):
    """dB with the mask that the dA+dR kernel leaves equals dB that hashes for itself, bit for bit, and the oracle."""
    from cute_mma_b200 import _functional as F
    N, gs, rs, dt, act = 192, 64, 8, torch.bfloat16, "silu_gate"
    A, B, R, dC = _inputs(M, K, N, gs, rs, dt, 11)
    bias = torch.randn(N // gs, K, device=DEV).to(dt) if ib else None
    seeds = torch.randint(1, 1 << 62, (N // gs,), dtype=torch.int64, device=DEV)
    dA, dR, dB, _ = cp.backward(dC, A, B, R, gs, rs, activation=act, internal_bias=bias, dropout_seeds=seeds, dropout_p=p)
    own = F._backward_db(dC, A, R, gs, rs, 1, internal_bias=bias, dropout_seeds=seeds, dropout_p=p)
    cp.check_device_status()
    assert torch.equal(dB, own)
    f = [t.float() for t in (A, B, R)]
    kw = dict(internal_bias=None if bias is None else bias.float(), dropout_seeds=seeds, dropout_p=p)
    ref = O.prism_backward(dC.float(), *f, gs, rs, act, **kw)
    C, _ = cp.forward(A, B, R, gs, rs, activation=act, internal_bias=bias, dropout_seeds=seeds, dropout_p=p, training=True)
    assert O.rel_err(C.float(), O.prism_forward(*f, gs, rs, act, **kw)) < TOL
    for got, r in zip((dA, dR, dB), ref):
        assert O.rel_err(got.float(), r) < TOL


@pytest.mark.parametrize("M,K,G,gs", [(1, 64, 12, 96), (100, 72, 9, 96), (300, 520, 7, 128), (1000, 264, 3, 512)])
@pytest.mark.parametrize("opts", ["plain", "gate", "ib", "drop"])
def test_group_parts_of_dadr(M, K, G, gs, opts):
    """Few tiles: the groups split over CTA pairs against one part (a plan given by hand is never split) and the oracle.
    A group's dR does not depend on the split; dA's partial sums meet in fp32."""
    from cute_mma_b200 import _functional as F
    from cute_mma_b200 import _lib
    N, rs, dt = G * gs, 8, torch.bfloat16
    act, gate = (None, 0) if opts == "plain" else ("silu_gate", 1)
    A, B, R, dC = _inputs(M, K, N, gs, rs, dt, 13)
    ib = torch.randn(G, K, device=DEV).to(dt) if opts == "ib" else None
    kw = dict(dropout_seeds=torch.arange(1, G + 1, device=DEV), dropout_p=0.25) if opts == "drop" else {}
    before = _lib.lib().prism_launch_count()
    got = F._backward_dadr(dC, A, B, R, gs, rs, gate, internal_bias=ib, **kw)
    n_split = _lib.lib().prism_launch_count() - before
    one = F._backward_dadr(dC, A, B, R, gs, rs, gate, internal_bias=ib, tile_cfg=[0, -1, 0], **kw)
    n_one = _lib.lib().prism_launch_count() - before - n_split
    cp.check_device_status()
    assert n_split == n_one + 1, "this shape is meant to be split"
    ref = O.prism_backward(dC.float(), A.float(), B.float(), R.float(), gs, rs, act,
                           internal_bias=None if ib is None else ib.float(), **kw)
    assert torch.equal(got[1], one[1]) and (ib is None or torch.equal(got[2], one[2]))
    assert O.rel_err(got[0].float(), one[0].float()) < 2 ** -8 + 1e-3    # one rounding to bf16 on either side
    assert O.rel_err(got[0].float(), ref[0]) < TOL and O.rel_err(got[1].float(), ref[1]) < TOL
