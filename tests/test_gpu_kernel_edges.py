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


@pytest.mark.parametrize("M,K,N,gs,part_rows", [(128, 256, 256, 256, 0),           # one token block: never split
                                                (129, 272, 512, 256, 0),           # two blocks, features past the first pair
                                                (2200, 256, 256, 128, 9 * 256),    # few tiles: split as often as it pays
                                                (4096, 1024, 4096, 256, 0),        # 64 tiles: one wave, not split
                                                (1300, 1008, 5120, 256, 9 * 512)]) # 80 tiles: two rows of the last wave are
@pytest.mark.parametrize("out", [None, torch.float32])
def test_split_plan_of_db(M, K, N, gs, part_rows, out):
    """The plan, as the rows of fp32 partial sums it asks for (74 CTA pairs), and its dB against the unsplit one and the oracle."""
    from cute_mma_b200 import _functional as F
    from cute_mma_b200 import _lib
    rs, dt, act = 16, torch.bfloat16, "sigmoid_gate"
    if torch.cuda.get_device_properties(0).multi_processor_count == 148:
        assert _lib.lib().prism_workspace_bytes(2, M, N, K, gs, rs, 1, None) == 256 + (part_rows * K * 4 + 255) // 256 * 256
    A, B, R, dC = _inputs(M, K, N, gs, rs, dt, 9)
    dB = cp.backward(dC, A, B, R, gs, rs, activation=act, dB_dtype=out)[2]
    one = F._backward_db(dC, A, R, gs, rs, 2, out_dtype=out, tile_cfg=[0, -1])
    cp.check_device_status()
    ref = O.prism_backward(dC.float(), A.float(), B.float(), R.float(), gs, rs, act)[2]
    assert dB.dtype == (out or dt) and O.rel_err(dB.float(), ref) < TOL
    # fp32 sums of at most 2200 products in another order; bf16: each side rounds by up to 2^-8, so that values on two sides
    # of a rounding boundary end one unit in the last place, 2^-7, apart
    assert torch.equal(dB, one) if part_rows == 0 else O.rel_err(dB.float(), one.float()) < (1e-5 if out else 2 ** -7 + 1e-5)


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
    need = _lib.lib().prism_workspace_bytes
    assert need(1, M, N, K, gs, rs, 1, None) > need(1, M, N, K, gs, rs, 1, F._cfg_array([0, -1, 0])), "this shape is meant to be split"
    got = F._backward_dadr(dC, A, B, R, gs, rs, gate, internal_bias=ib, **kw)
    one = F._backward_dadr(dC, A, B, R, gs, rs, gate, internal_bias=ib, tile_cfg=[0, -1, 0], **kw)
    cp.check_device_status()
    ref = O.prism_backward(dC.float(), A.float(), B.float(), R.float(), gs, rs, act,
                           internal_bias=None if ib is None else ib.float(), **kw)
    assert torch.equal(got[1], one[1]) and (ib is None or torch.equal(got[2], one[2]))
    assert O.rel_err(got[0].float(), one[0].float()) < 2 ** -8 + 1e-3    # one rounding to bf16 on either side
    assert O.rel_err(got[0].float(), ref[0]) < TOL and O.rel_err(got[1].float(), ref[1]) < TOL


class _Seen(torch.utils._python_dispatch.TorchDispatchMode):
    """Runs every op as it comes and remembers the package's own."""

    def __init__(self):
        super().__init__()
        self.ops = set()

    def __torch_dispatch__(self, func, types, args=(), kwargs=None):
        if func.namespace == "prism_b200":
            self.ops.add(func.__name__)
        return func(*args, **(kwargs or {}))


@pytest.mark.parametrize("kw", [dict(), dict(bias=False, reconn_sz=16), dict(reconn_sz=32), dict(cayley_order=2),
                                dict(activation="silu_gate", internal_bias=True), dict(activation="sigmoid_gate", ar_scale_init=0.7),
                                dict(activation="silu_gate", dropout=0.2, internal_bias=True),
                                dict(activation="silu_gate", input_shuffle=True, reconn_sz=16, internal_bias=True),
                                dict(input_shuffle=True, reconn_sz=16)])
@pytest.mark.parametrize("train_weight", [False, True])
def test_eager_layer_is_the_custom_ops(kw, train_weight):
    """An ordinary call runs as one autograd node, a call under a dispatch mode as the custom ops: the same numbers, the
    same gradients, for a strided 3-D input and a strided output gradient, twice through a retained graph."""
    from cute_mma_b200 import _module
    K, N, dt = 192, 256, torch.bfloat16
    torch.manual_seed(1)
    layer = cp.PrismLinear(K, N, **{"group_size": 64, "reconn_sz": 8, **kw})
    if not layer.activation:
        torch.nn.init.normal_(layer.reconn, 0.0, 0.1)
    layer = layer.to(DEV).to(dt).train()
    layer.weight.requires_grad_(train_weight)
    x0 = torch.randn(5, 2 * K, 34, device=DEV).to(dt)
    dy = torch.randn(N, 5, 34, device=DEV).to(dt).permute(1, 2, 0)
    res = []
    for mode in (None, _Seen()):
        x = x0[:, ::2].transpose(1, 2).detach().requires_grad_()
        layer.zero_grad(set_to_none=True)
        torch.manual_seed(2)   # dropout seeds
        if mode is None:
            assert _module._plain_eager(x, layer.weight)
            y = layer(x)
            y.backward(dy, retain_graph=True)
            y.backward(dy)
        else:
            with mode:
                assert not _module._plain_eager(x, layer.weight)
                y = layer(x)
                y.backward(dy, retain_graph=True)
                y.backward(dy)
            assert "forward.default" in mode.ops
        res.append([y.detach(), x.grad] + [p.grad for p in layer.parameters()])
    with torch.no_grad():
        torch.manual_seed(2)
        assert torch.equal(layer(x0[:, ::2].transpose(1, 2)), res[0][0])
    cp.check_device_status()
    assert (res[0][2] is None) == (not train_weight)
    for a, b in zip(*res):
        assert (a is None and b is None) or torch.equal(a, b)


def test_eager_layer_under_autograd_features():
    from cute_mma_b200 import _module
    K, N, dt = 128, 128, torch.float16
    layer = cp.PrismLinear(K, N, group_size=64, reconn_sz=8, activation="silu_gate").to(DEV).to(dt)
    x = torch.randn(16, K, device=DEV, dtype=dt, requires_grad=True)
    w = layer.weight
    # what has to see the ops is not taken
    with torch.device(DEV):                       # a function mode
        assert not _module._plain_eager(x, w)
    with torch.autograd.forward_ad.dual_level():
        assert not _module._plain_eager(x, w)
    torch.func.vmap(lambda t: (lambda _: t)(_flag(_module, t)))(x.detach())
    assert not _module._plain_eager(x.cpu()) and not _module._plain_eager(torch.nn.Buffer(x.detach()).as_subclass(_Sub))
    # saved-tensor hooks see what is kept; nothing is kept where no gradient is wanted
    packed = []
    with torch.autograd.graph.saved_tensors_hooks(lambda t: packed.append(t) or t.clone(), lambda t: t):
        y = layer(x)
    assert len(packed) >= 3
    g1, = torch.autograd.grad(y.float().sum(), x, create_graph=True)
    with pytest.raises(RuntimeError):             # no second derivative, and no silent zero either
        g1.float().pow(2).sum().backward()
    layer.requires_grad_(False)
    assert not layer(x.detach()).requires_grad
    g2, = torch.autograd.grad(layer(x).float().sum(), x)
    assert torch.equal(g1, g2)
    cp.check_device_status()


@pytest.mark.parametrize("kw", [dict(activation="silu_gate", internal_bias=True), dict(),
                                dict(activation="silu_gate", input_shuffle=True, reconn_sz=16, internal_bias=True)])
def test_backward_of_an_ordinary_forward_by_other_means(kw):
    """A dispatch mode around the backward sees the custom ops; a batch of output gradients is taken one by one: the
    gradients of the ordinary backward."""
    K, N, dt = 128, 256, torch.bfloat16
    torch.manual_seed(3)
    layer = cp.PrismLinear(K, N, **{"group_size": 64, "reconn_sz": 8, **kw}).to(DEV).to(dt)
    torch.nn.init.normal_(layer.reconn, 0.0, 0.1)
    x = torch.randn(40, K, device=DEV, dtype=dt, requires_grad=True)
    dy = torch.randn(3, 40, N, device=DEV, dtype=dt)
    wanted = [x] + [p for p in layer.parameters() if p.requires_grad]
    y = layer(x)
    plain = [torch.autograd.grad(y, wanted, d, retain_graph=True) for d in dy]
    mode = _Seen()
    with mode:
        seen = torch.autograd.grad(y, wanted, dy[0], retain_graph=True)
    assert "backward.default" in mode.ops and "forward.default" not in mode.ops
    batched = torch.autograd.grad(y, wanted, dy, is_grads_batched=True)
    cp.check_device_status()
    for i, b in enumerate(batched):
        assert torch.equal(seen[i], plain[0][i]) and torch.equal(b, torch.stack([p[i] for p in plain]))


@pytest.mark.parametrize("kw", [dict(activation="silu_gate", internal_bias=True), dict()])   # the second: Cayley
def test_unpacked_views_of_another_layout(kw):
    """Saved-tensor hooks that hand back every second element of a wider buffer: the gradients of the plain call."""
    K, N, dt = 128, 256, torch.bfloat16
    layer = cp.PrismLinear(K, N, group_size=64, reconn_sz=8, **kw).to(DEV).to(dt)
    torch.nn.init.normal_(layer.reconn, 0.0, 0.1)
    x = torch.randn(40, K, device=DEV, dtype=dt, requires_grad=True)
    dy = torch.randn(40, N, device=DEV, dtype=dt)
    wanted = [x] + [p for p in layer.parameters() if p.requires_grad]
    plain = torch.autograd.grad(layer(x), wanted, dy)
    with torch.autograd.graph.saved_tensors_hooks(lambda t: torch.stack((t, -t), -1), lambda s: s[..., 0]):
        y = layer(x)
    got = torch.autograd.grad(y, wanted, dy)
    cp.check_device_status()
    assert all(torch.equal(a, b) for a, b in zip(plain, got))


@pytest.mark.parametrize("grad", [False, True])
def test_views_with_the_negative_bit(grad):
    """Values that are the negative of what lies in memory: operands and output gradients alike."""
    K, N, gs, rs, dt = 128, 256, 64, 8, torch.float16
    A, B, R, dC = _inputs(40, K, N, gs, rs, dt, 25)
    A.requires_grad_(grad)
    y = cp.prism_linear(A, B, R, group_size=gs, reconn_sz=rs, activation="silu_gate")
    flipped = torch._neg_view(-A)
    assert flipped.is_neg()
    assert torch.equal(cp.prism_linear(flipped, B, R, group_size=gs, reconn_sz=rs, activation="silu_gate"), y)
    if grad:
        g, = torch.autograd.grad(y, A, dC, retain_graph=True)
        assert torch.equal(torch.autograd.grad(y, A, torch._neg_view(-dC))[0], g)
    cp.check_device_status()


class _Sub(torch.Tensor):
    pass


def _flag(module, t):
    assert not module._plain_eager(t)
    return t


@pytest.mark.parametrize("K,rs", [(8, 8), (1032, 8), (1040, 16)])   # one thread; past 1024 columns, a row of two blocks
def test_reductions_of_dadr_share_a_launch(K, rs):
    """dR (16 and 32 bits), the internal-bias gradient and dA of split groups, with extra pairs and without."""
    from cute_mma_b200 import _functional as F
    M, G, gs, dt, act = 700, 6, 128, torch.bfloat16, "silu_gate"
    A, B, R, dC = _inputs(M, K, G * gs, gs, rs, dt, 17)
    ib = torch.randn(G, K, device=DEV).to(dt)
    ref = O.prism_backward(dC.float(), A.float(), B.float(), R.float(), gs, rs, act, internal_bias=ib.float())
    for cfg in (None, [1, 1, 1], [3, -1, 0]):
        dA, dR, dib = F._backward_dadr(dC, A, B, R, gs, rs, 1, internal_bias=ib, tile_cfg=cfg, dR_dtype=torch.float32)
        dA2, dR2, dib2 = F._backward_dadr(dC, A, B, R, gs, rs, 1, internal_bias=ib, tile_cfg=cfg)
        cp.check_device_status()
        assert torch.equal(dA, dA2) and torch.equal(dib, dib2) and torch.equal(dR.to(dt), dR2)
        assert O.rel_err(dA.float(), ref[0]) < TOL and O.rel_err(dR, ref[1]) < TOL and O.rel_err(dib.float(), ref[3]) < TOL


@pytest.mark.parametrize("M,path", [(1, 2), (100, 2), (100, 1), (700, 1)])    # the streaming kernel and the general one
@pytest.mark.parametrize("K", [8, 72, 136, 1000])                             # one block; odd counts of blocks; a ragged chunk
@pytest.mark.parametrize("act", [None, "silu_gate"])
def test_rotations_of_8_are_widened_in_the_forward(M, K, path, act):
    """More chunks than stages and more tiles than CTA pairs; non-finite values in one block reach that block only."""
    gs, rs, dt = 128, 8, torch.bfloat16
    N = gs * (200 if K < 100 else 600 if M == 700 else 9)   # the last: long enough for the copy
    A, B, R, _ = _inputs(M, K, N, gs, rs, dt, 19)
    C, _ = cp.forward(A, B, R, gs, rs, activation=act, tile_cfg=[0, 0, 0, path])
    cp.check_device_status()
    assert O.rel_err(C.float(), O.prism_forward(A.float(), B.float(), R.float(), gs, rs, act)) < TOL
    R[:8, :8] = float("inf")                     # the first block of group 0
    C2, _ = cp.forward(A, B, R, gs, rs, activation=act, tile_cfg=[0, 0, 0, path])
    assert torch.equal(C2[:, gs:], C[:, gs:])


@pytest.mark.parametrize("M,N,gs", [(1, 256, 256), (257, 1024, 256), (256, 18944, 256), (300, 768, 192), (64, 512, 512)])
def test_tile_width_of_short_forwards(M, N, gs):
    """Narrow tiles while they fit one wave (74 tiles of 256: none; groups of 192: 64 wide) give the bits of wide ones."""
    K, rs, dt = 200, 8, torch.float16
    A, B, R, _ = _inputs(M, K, N, gs, rs, dt, 21)
    bias = torch.randn(N, device=DEV).to(dt)
    C, _ = cp.forward(A, B, R, gs, rs, activation="silu_gate", bias=bias, tile_cfg=[0, 0, 0, 1])
    wide, _ = cp.forward(A, B, R, gs, rs, activation="silu_gate", bias=bias, tile_cfg=[192 if gs == 192 else 256, 0, 0, 1])
    cp.check_device_status()
    assert torch.equal(C, wide)
    assert O.rel_err(C.float(), O.prism_forward(A.float(), B.float(), R.float(), gs, rs, "silu_gate", bias=bias.float())) < TOL


@pytest.mark.parametrize("M", [128, 700])                                        # bf16 silu: stores by TMA; plain ones below 256
@pytest.mark.parametrize("gs,N", [(16, 48), (32, 64), (96, 192), (256, 512)])   # stores of 16, 32 and 64 rows of dB
@pytest.mark.parametrize("K", [8, 72, 200, 328])                                 # features that end inside a 64-wide store
@pytest.mark.parametrize("rs,dt,gate", [(8, torch.bfloat16, 1), (16, torch.bfloat16, 1), (16, torch.float16, 2)])
def test_transposed_stores_of_db(gs, N, K, M, rs, dt, gate):
    """16-bit dB is the rounded fp32 dB, which leaves by plain stores, and touches nothing beside it."""
    from cute_mma_b200 import _functional as F
    K -= K % rs if K > rs else K - rs
    A, B, R, dC = _inputs(M, K, N, gs, rs, dt, 23)
    pad = torch.full((N + 2, K), 7.0, dtype=dt, device=DEV)
    dB = F._backward_db(dC, A, R, gs, rs, gate, dc_scale=0.5, dB_out=pad[1:N + 1], tile_cfg=[0, -1])
    wide = F._backward_db(dC, A, R, gs, rs, gate, dc_scale=0.5, out_dtype=torch.float32, tile_cfg=[0, -1])
    cp.check_device_status()
    assert torch.equal(dB, wide.to(dt)) and (pad[0] == 7).all() and (pad[N + 1] == 7).all()
    ref = O.prism_backward(0.5 * dC.float(), A.float(), B.float(), R.float(), gs, rs, (None, "silu_gate", "sigmoid_gate")[gate])[2]
    assert O.rel_err(wide, ref) < TOL
