"""Products on single SMs with narrow tiles (csrc/gemm_narrow.cu) against float64: the edges of its tiles, its epilogues, its refusals."""
import math

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.fixture(scope="module")
def fast():
    from leone_b200.ops.cuda import CudaOps
    ops = CudaOps(DEV, torch.bfloat16)
    ops.bind_status(torch.zeros(4, dtype=torch.int32, device=DEV))
    return ops.fast


def _run(fast, x, w, out, epilogue, residual, width, norm=(None, 0, 0.0), bias=None):
    m, k = x.shape
    return fast.calls.leone_gemm_narrow(x, w, out, residual, m, w.shape[0], k, x.stride(0), w.stride(0), out.stride(0), epilogue, width,
                                        fast.status, fast.sm_count, *norm, None, bias, fast._stream())


def _close(got, want, rel, floor):
    # bf16 outputs: half a unit in the last place; fp32 ones: sums of k terms in any order (4 sqrt(k) eps of a term's size)
    err = (got.double() - want).abs()
    assert bool((err <= rel * want.abs() + floor).all()), float((err - rel * want.abs()).max())


# one token; rows that are no multiple of 8; a whole tile and one more; last tiles of weights of one row and of eight; K of one
# k-block, of a ragged one, and longer than the ring; one tile a block and several
@pytest.mark.parametrize("m,n,k,width", [(1, 16, 64, 16), (7, 161, 136, 32), (33, 2048, 2048, 16), (64, 4104, 1024, 32),
                                                (77, 2048, 6144, 16), (128, 520, 520, 64), (129, 264, 64, 48), (200, 3072, 2048, 64),
                                                (300, 1040, 4096, 128), (640, 2064, 1000, 256), (40, 20000, 256, 32)])
def test_every_epilogue_against_float64(fast, m, n, k, width):
    g = torch.Generator(device=DEV).manual_seed(m + n + k)
    x = torch.randn((m, k), device=DEV, generator=g).to(torch.bfloat16)
    w = (torch.randn((n, k), device=DEV, generator=g) * 0.05).to(torch.bfloat16)
    want = x.double() @ w.double().t()
    floor = 4 * math.sqrt(k) * 2 ** -23 * 4
    bias = torch.randn(n + 16, device=DEV, generator=g)[:n]
    out = torch.full((m, n), 9.0, device=DEV, dtype=torch.bfloat16)
    assert _run(fast, x, w, out, 0, None, width) == 0
    _close(out, want, 2 ** -8, floor)
    assert _run(fast, x, w, out, 0, None, width, bias=bias) == 0
    _close(out, want + bias.double(), 2 ** -8, floor)
    out32 = torch.full((m, n), 9.0, device=DEV)
    assert _run(fast, x, w, out32, 1, None, width) == 0
    _close(out32, want, 1e-5, floor)
    res = torch.randn((m, n), device=DEV, generator=g)
    hidden = res.clone()
    assert _run(fast, x, w, hidden, 2, hidden, width) == 0
    _close(hidden, want + res.double(), 1e-5, floor)
    again = res.clone()
    assert _run(fast, x, w, again, 2, again, width) == 0 and torch.equal(hidden, again)
    ss = torch.rand((3, m), device=DEV, generator=g) * k
    rs = torch.rsqrt(ss.double().sum(0)[:, None] / k + 1e-6)
    assert _run(fast, x, w, out32, 1, None, width, (ss, 3, 1e-6)) == 0
    _close(out32, want * rs, 1e-5, floor)
    if width % 32 == 0 and n >= 32:
        inter = n // 32 * 16
        act = torch.full((m, inter), 9.0, device=DEV, dtype=torch.bfloat16)
        assert _run(fast, x, w[:2 * inter], act, 3, None, width) == 0
        pairs = want[:, :2 * inter].view(m, -1, 2, 16)
        gate, up = pairs[:, :, 0].reshape(m, inter), pairs[:, :, 1].reshape(m, inter)
        _close(act, gate * torch.sigmoid(gate) * up, 2 ** -7, 1e-4)
    torch.cuda.synchronize()
    assert int(fast.status.abs().sum()) == 0


def test_rows_that_a_vector_cannot_take(fast):
    """Outputs whose rows start anywhere are written element by element; their neighbours stay."""
    x = torch.randn((50, 128), device=DEV).to(torch.bfloat16)
    w = torch.randn((45, 128), device=DEV).to(torch.bfloat16)
    want = x.double() @ w.double().t()
    for dtype, epilogue, rel in ((torch.bfloat16, 0, 2 ** -8), (torch.float32, 1, 1e-5)):
        wide = torch.full((50, 51), 7.0, device=DEV, dtype=dtype)
        assert _run(fast, x, w, wide[:, 3:48], epilogue, None, 32) == 0
        _close(wide[:, 3:48], want, rel, 1e-4)
        assert bool((wide[:, :3] == 7).all()) and bool((wide[:, 48:] == 7).all())


def test_refusals(fast):
    x = torch.zeros((8, 64), device=DEV, dtype=torch.bfloat16)
    w = torch.zeros((64, 64), device=DEV, dtype=torch.bfloat16)
    out = torch.zeros((8, 64), device=DEV, dtype=torch.bfloat16)
    for width in (8, 24, 272):
        assert _run(fast, x, w, out, 0, None, width) < 0
    assert _run(fast, x, w, out, 2, None, 32) < 0 and _run(fast, x, w, out, 3, None, 48) < 0


@pytest.mark.parametrize("m,n,k,epilogue", [(33, 2048, 2048, 0), (128, 1000, 520, 2), (77, 1024, 2048, 3), (129, 45, 128, 0), (300, 2080, 1024, 3),
                                            (257, 1016, 2048, 1), (1027, 2048, 512, 2)])
def test_the_rules_forms_agree(fast, m, n, k, epilogue):
    """What the rules for products without a norm choose, against the forms that they replace and float64."""
    g = torch.Generator(device=DEV).manual_seed(m * n)
    x = torch.randn((m, k), device=DEV, generator=g).to(torch.bfloat16)
    w = (torch.randn((n, k), device=DEV, generator=g) * 0.05).to(torch.bfloat16)
    want = x.double() @ w.double().t()
    start = torch.randn((m, n), device=DEV, generator=g)
    if epilogue == 2:
        want = want + start.double()
    if epilogue == 3:
        pairs = want.view(m, -1, 2, 16)
        gate, up = pairs[:, :, 0].reshape(m, -1), pairs[:, :, 1].reshape(m, -1)
        want = gate * torch.sigmoid(gate) * up
    outs = []
    for narrow in (True, False):
        fast.use_narrow = narrow
        out = start.clone() if epilogue == 2 else torch.empty((m, n // 2 if epilogue == 3 else n), device=DEV,
                                                               dtype=torch.float32 if epilogue == 1 else torch.bfloat16)
        assert fast._gemm(x, w, out, epilogue, out if epilogue == 2 else None, n)
        outs.append(out)
    fast.use_narrow = True
    rel = {0: 2 ** -8, 1: 1e-5, 2: 1e-5, 3: 2 ** -7}[epilogue]
    for out in outs:
        _close(out, want, rel, 4 * math.sqrt(k) * 2 ** -23 * 4 if epilogue != 3 else 1e-4)
