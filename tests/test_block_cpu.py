"""The decoder block in one native call, without a GPU: what its autograd function saves and what it takes back, over a stand-in for the library."""
import ctypes
import gc

import pytest
import torch

from tesseract_b200.ops import block

SHAPE = (2, 3, 128, 2, 1, 64, 264)          # B, S, W, H, Hkv, D, F
PACKED = 4 * 64


class Library:
    """Entry points that note the addresses they are given."""

    def tsb_block_bytes(self, shape, has_res, sizes):
        sizes[:] = [4096, 8192, 512, 256]
        return 0

    def tsb_block_forward(self, shape, p, f, causal, stream):
        self.forward = list(p)
        return 0

    def tsb_block_backward_down(self, shape, p, stream):
        return 0

    def tsb_block_backward(self, shape, p, f, has_res, causal, stream):
        return 0


@pytest.fixture
def library(monkeypatch):
    fake = Library()
    monkeypatch.setattr(block, "lib", lambda: fake)
    monkeypatch.setattr(block, "stream_ptr", lambda device: 0)
    return fake


def _call(has_res=True, given=True):
    B, S, W, H, Hkv, D, F = SHAPE
    shapes = [(W,), (W, W), (Hkv * D, W), (Hkv * D, W), (W, W), (W,), (F, W), (F, W), (W, F)]
    flat = torch.randn(sum(a[0] * (a[1] if len(a) > 1 else 1) for a in shapes)).bfloat16()
    grad, at, params = torch.zeros_like(flat), 0, []
    for s in shapes:
        n = s[0] * (s[1] if len(s) > 1 else 1)
        p = torch.nn.Parameter(torch.empty(0, dtype=torch.bfloat16))
        p.data = flat[at:at + n].view(s)
        p.main_grad = grad[at:at + n].view(s)
        params.append(p)
        at += n
    own = [params[i] for i in (0, 1, 4, 5, 6, 8)]
    behind = [params[i] for i in (2, 3, 7)]
    behind = behind + [p.main_grad for p in behind] if given else None
    x = torch.randn(B, S, W).bfloat16().requires_grad_()
    res = torch.randn(B, S, W).bfloat16().requires_grad_() if has_res else None
    tables = torch.zeros(8, D // 2), torch.zeros(8, D // 2)
    out = block.decoder_block(x, res, own, [p.main_grad for p in own], *tables, SHAPE, (1e-5, 1e-5, 0.125), True, behind)
    return params, x, res, out


def _at(address, n, dtype=torch.bfloat16):
    return torch.frombuffer((ctypes.c_char * (n * dtype.itemsize)).from_address(address), dtype=dtype)


def _noted(library, has_res=True, given=True, **around):
    """Weights and what the backward call finds at the addresses of the stacks, while it runs."""
    with torch.autograd.graph.saved_tensors_hooks(around["pack"], around["unpack"]):
        params, x, res, (out, res2) = _call(has_res, given)
    seen = {}

    def down(shape, p, stream):
        assert all(v % 16 == 0 for v in p)
        seen.update(down=_at(p[0], 128 * 264).clone().view(128, 264), first=list(p))
        return 0

    def backward(shape, p, f, has_res, causal, stream):
        assert all(v % 16 == 0 for v in p)
        seen.update(qkv=_at(p[2], PACKED * 128).clone().view(PACKED, 128), gate_up=_at(p[5], 528 * 128).clone().view(528, 128), p=list(p))
        return 0

    library.tsb_block_backward_down, library.tsb_block_backward = down, backward
    torch.autograd.backward([out, res2], [torch.zeros_like(out), torch.zeros_like(res2)])
    return params, seen


@pytest.mark.parametrize("has_res,given", [(True, True), (False, True), (True, False)])
def test_saved_are_whole_stacks(library, has_res, given):
    """A hook that moves what is saved (activations kept on the host do) moves all rows of q / k / v and of gate / up. The stacks as saved, without a
    look at memory: what is behind a copy of the first matrix is not this program's."""
    kept = []

    def pack(t):
        kept.append(t.detach().clone())
        return kept[-1]

    with torch.autograd.graph.saved_tensors_hooks(pack, lambda t: t):
        params, *_ = _call(has_res, given)
    for p in params:
        assert any(t.shape == p.shape and torch.equal(t, p.detach()) for t in kept)
    params, seen = _noted(library, has_res, given, pack=pack, unpack=lambda t: t)
    assert torch.equal(seen["qkv"], torch.cat([p.detach() for p in params[1:4]]))
    assert torch.equal(seen["gate_up"], torch.cat([p.detach() for p in params[6:8]]))
    assert seen["p"][11] == params[1].main_grad.data_ptr() and seen["p"][14] == params[6].main_grad.data_ptr()
    assert seen["first"][2] == params[8].main_grad.data_ptr()
    assert library.forward[3] not in (seen["p"][2], seen["p"][5])


def test_nothing_is_copied_without_hooks(library):
    params, seen = _noted(library, pack=lambda t: t, unpack=lambda t: t)
    assert seen["p"][2] == params[1].data_ptr() and seen["p"][5] == params[6].data_ptr() and seen["first"][0] == params[8].data_ptr()


@pytest.mark.parametrize("keep", [False, True])
def test_widest_activations_are_let_go_halfway(library, keep):
    """Between the two calls of a backward pass, unless the graph is kept for another one."""
    _, x, _, (out, _) = _call()
    size, seen = 8192, []

    def backward(shape, p, f, has_res, causal, stream):
        gc.collect()
        seen.append(any(t.dtype is torch.uint8 and t.numel() == size for t in gc.get_objects() if type(t) is torch.Tensor) or _saved(out))
        return 0

    def _saved(out):
        try:
            return any(t.numel() == size for t in out.grad_fn.saved_tensors)
        except RuntimeError:                              # (let go)
            return False

    library.tsb_block_backward = backward
    out.backward(torch.zeros_like(out), retain_graph=keep)
    if keep:
        out.backward(torch.zeros_like(out))
    assert seen == ([True, False] if keep else [False])


def test_saved_come_back_off_sixteen_bytes_or_strided(library):
    def unpack(t):
        wide = torch.empty(t.numel() + 1, dtype=t.dtype)[1:].view(t.shape).copy_(t)
        return wide if t.dim() != 2 else wide.t().contiguous().t()

    params, seen = _noted(library, pack=lambda t: t.detach().clone(), unpack=unpack)
    assert torch.equal(seen["qkv"], torch.cat([p.detach() for p in params[1:4]]))
    assert torch.equal(seen["gate_up"], torch.cat([p.detach() for p in params[6:8]]))
    assert torch.equal(seen["down"], params[8].detach())


@pytest.mark.parametrize("spoil", [lambda t: t[:1], lambda t: t.double()])
def test_saved_come_back_as_something_else(library, spoil):
    with torch.autograd.graph.saved_tensors_hooks(lambda t: t, lambda t: spoil(t) if t.shape == (128, 264) else t):
        _, _, _, (out, _) = _call()
    library.tsb_block_backward_down = None                # (not reached)
    with pytest.raises(RuntimeError, match="saved tensor"):
        out.backward(torch.zeros_like(out))
