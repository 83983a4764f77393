"""The layer object reads its weights where the caller keeps them, on every call."""
import pytest
import torch

from oracle import moe_oracle as O
from tilelang_moe_b200 import kernels, ops

pytestmark = pytest.mark.gpu
NAMES = ["router_weight", "shared_gate", "shared_up", "shared_down", "routed_gate", "routed_up", "routed_down"]


def _layer(H, I, E, T, k=2):
    return kernels.FusedMoETileLang(H, I, E, 1, k, 1, T, dtype=torch.bfloat16)


def _inputs(cuda, T, H, I, E, seed, k=2):
    x, w = O.make_fusedmoe_inputs(1, T, H, I, E, 1, k, dtype=torch.bfloat16, seed=seed)
    return x.to(cuda), [w[n].to(cuda) for n in NAMES]


def _two_streams(x, w, H, I, E, T, k=2):
    m = _layer(H, I, E, T, k)
    m.STACK_LIMIT_BYTES = 0                       # the shared expert as a GEMM of its own
    return m.forward(x, *w)


@pytest.mark.parametrize("T", [5, 300])
def test_a_write_to_a_weight_is_seen(cuda, lib, T):
    H, I, E = 256, 128, 8
    x, w = _inputs(cuda, T, H, I, E, 1)
    _, w2 = _inputs(cuda, T, H, I, E, 2)
    m = _layer(H, I, E, T)
    m.forward(x, *w)
    for i in range(1, 7):
        w[i].data.copy_(w2[i])                    # leaves the version counter of w[i] alone
        assert torch.equal(m.forward(x, *w), _two_streams(x, w, H, I, E, T)), NAMES[i]
    ops.check_status(cuda)


def test_other_weights_at_the_same_addresses(cuda, lib):
    T, H, I, E = 64, 256, 128, 8
    x, w = _inputs(cuda, T, H, I, E, 3)
    m = _layer(H, I, E, T)
    first = m.forward(x, *w).clone()
    host = [t.cpu().flip(0) for t in w]
    at = {t.data_ptr() for t in w}
    del w
    w = [t.to(cuda) for t in host]                # the caching allocator hands the blocks out again
    assert at & {t.data_ptr() for t in w}
    y = m.forward(x, *w)
    assert torch.equal(y, _two_streams(x, w, H, I, E, T)) and not torch.equal(y, first)
    ops.check_status(cuda)


def test_weights_the_gemms_cannot_read_in_place(cuda, lib):
    """Transposed views, storage off the 16-byte boundary, a leading dimension of one, another type of the shared expert:
    taken through a copy of their own on every call."""
    T, H, I, E = 40, 128, 64, 4
    x, w = _inputs(cuda, T, H, I, E, 4)
    want = _two_streams(x, w, H, I, E, T).clone()

    def off(t):                                   # the same values two bytes past a boundary
        base = torch.empty(t.numel() + 1, dtype=t.dtype, device=t.device)
        base[1:].copy_(t.flatten())
        return base[1:].view(t.shape)

    turned = [t.mT.contiguous().mT if t.dim() > 1 else t for t in w]
    for name, forms in (("strided", turned), ("off", [w[0], *map(off, w[1:])]),
                        ("ones", [w[0], *(t[None].clone() for t in w[1:4]), *w[4:]]), ("float", [w[0], *(t.float() for t in w[1:4]), *w[4:]])):
        forms[0] = w[0]
        m = _layer(H, I, E, T)
        assert torch.equal(m.forward(x, *forms), want), name
        forms[1].data.mul_(0.5)
        w_half = [w[0], w[1] * 0.5, *w[2:]]
        assert torch.equal(m.forward(x, *forms), _two_streams(x, w_half, H, I, E, T)), name
    with pytest.raises(RuntimeError):             # shapes that do not belong together stay refused
        _layer(H, I, E, T).forward(x, w[0], w[1][:-8], *w[2:])
    with pytest.raises(RuntimeError):
        _layer(H, I, E, T).forward(x, *w[:5], w[5].mT.contiguous(), w[6])
    ops.check_status(cuda)


@pytest.mark.parametrize("T,E,k,H,I", [(4095, 8, 2, 1024, 128), (4096, 8, 2, 1024, 256), (4097, 8, 2, 1024, 256), (1500, 2, 2, 2048, 512)])
def test_shared_group_on_large_batches(cuda, lib, T, E, k, H, I):
    """The shared expert as a group of its own tensor in the single-CTA and the CTA-pair kernel, on either side of the batch
    size up to which the kernels of a call are launched dependently."""
    x, w = _inputs(cuda, T, H, I, E, T, k)
    lg = ops.router_logits(x.view(-1, H), w[0])
    m = _layer(H, I, E, T, k)
    y = m.forward(x, *w, logits=lg)
    assert m._stack == (E + 1, I, H)
    n = _layer(H, I, E, T, k)
    n.STACK_LIMIT_BYTES = 0
    assert torch.equal(y, n.forward(x, *w, logits=lg)) and n._stack is None
    ref = O.fusedmoe(x.cpu(), *[t.cpu() for t in w], k, logits=lg.cpu())
    torch.testing.assert_close(y.float().cpu(), ref, rtol=1e-2, atol=2e-2)
    ops.check_status(cuda)


def test_as_many_experts_as_a_gemm_takes(cuda, lib):
    """1024 routed experts leave no group for the shared one: side-stream form, strided weights through copies as ever."""
    T, H, I, E = 6, 64, 8, 1024
    x, w = _inputs(cuda, T, H, I, E, 6)
    want = _two_streams(x, w, H, I, E, T).clone()
    turned = [w[0], *(t.mT.contiguous().mT for t in w[1:])]
    assert torch.equal(_layer(H, I, E, T).forward(x, *turned), want)
    ops.check_status(cuda)
