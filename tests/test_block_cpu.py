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

    def tsb_block_backward(self, shape, p, f, has_res, causal, part, stream):
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
    """Weights and what the backward call finds at their addresses, while it runs."""
    with torch.autograd.graph.saved_tensors_hooks(around["pack"], around["unpack"]):
        params, x, res, (out, res2) = _call(has_res, given)
    return params, _noted_after(library, out, res2)


def _noted_after(library, out, res2):
    seen = {"parts": []}

    def backward(shape, p, f, has_res, causal, part, stream):
        assert all(v % 16 == 0 for v in p)
        seen["parts"].append(part)
        if part == 1:
            seen.update(down=_at(p[6], 128 * 264).clone().view(128, 264), first=list(p))
        if part == 2:
            seen.update(qkv=_at(p[2], PACKED * 128).clone().view(PACKED, 128), gate_up=_at(p[5], 528 * 128).clone().view(528, 128), p=list(p))
        return 0

    library.tsb_block_backward = backward
    torch.autograd.backward([out, res2], [torch.zeros_like(out), torch.zeros_like(res2)])
    return seen


def _whole(params, seen):
    return (torch.equal(seen["qkv"], torch.cat([p.detach() for p in params[1:4]])) and torch.equal(seen["down"], params[8].detach())
            and torch.equal(seen["gate_up"], torch.cat([p.detach() for p in params[6:8]])))


@pytest.mark.parametrize("has_res,given", [(True, True), (False, True), (True, False)])
def test_stacks_are_whole_under_hooks(library, has_res, given):
    """A hook that moves what is saved (activations kept on the host do) leaves the weights alone: behind a copy of the first matrix of a stack
    would be memory that is not this program's."""
    kept = []

    def pack(t):
        kept.append(t.detach().clone())
        return kept[-1]

    with torch.autograd.graph.saved_tensors_hooks(pack, lambda t: t):
        params, *_ = _call(has_res, given)
    assert len(kept) == (3 if has_res else 4) and not any(t.shape == p.shape for t in kept for p in params)
    params, seen = _noted(library, has_res, given, pack=pack, unpack=lambda t: t)
    assert _whole(params, seen) and seen["parts"] == [1, 2]
    assert seen["p"][13] == params[1].main_grad.data_ptr() and seen["p"][16] == params[6].main_grad.data_ptr()
    assert seen["first"][17] == params[8].main_grad.data_ptr()


def test_nothing_is_copied_without_hooks(library):
    params, seen = _noted(library, pack=lambda t: t, unpack=lambda t: t)
    assert seen["p"][2] == params[1].data_ptr() and seen["p"][5] == params[6].data_ptr() and seen["first"][6] == params[8].data_ptr()


def test_storage_of_a_weight_exchanged_between_the_passes(library):
    """The weight as it is now, wherever it lies, as the modules take it."""
    params, x, res, (out, res2) = _call()
    for i in (2, 8):
        params[i].data = torch.empty(params[i].numel() + 1, dtype=torch.bfloat16)[1:].view(params[i].shape).copy_(params[i].detach())
    assert _whole(params, _noted_after(library, out, res2))


def test_storage_of_a_weight_exchanged_for_another_size(library):
    params, x, res, (out, res2) = _call()
    params[7].data = params[7].data[:8].clone()
    library.tsb_block_backward = None                     # (not reached)
    with pytest.raises(RuntimeError, match="came back"):
        out.backward(torch.zeros_like(out))


@pytest.mark.parametrize("i,refused", [(0, True), (4, True), (5, True), (8, True), (1, False), (2, False), (7, False)])
def test_weights_changed_in_place_between_the_passes(library, i, refused):
    """Norms, output and down projection refuse it, as their modules do; the stacks, which the modules take as views without a history, do not."""
    params, x, res, (out, res2) = _call()
    with torch.no_grad():
        params[i].add_(1)
    if refused:
        with pytest.raises(RuntimeError, match="inplace"):
            out.backward(torch.zeros_like(out))
    else:
        out.backward(torch.zeros_like(out))


@pytest.mark.parametrize("keep", [False, True])
def test_widest_activations_are_let_go_halfway(library, keep):
    """Between the two calls of a backward pass, unless the graph is kept for another one."""
    _, x, _, (out, _) = _call()
    size, seen = 8192, []

    def backward(shape, p, f, has_res, causal, part, stream):
        gc.collect()
        if part == 2:
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
        return wide if t.dim() != 3 else wide.transpose(1, 2).contiguous().transpose(1, 2)

    params, seen = _noted(library, has_res=False, pack=lambda t: t.detach().clone(), unpack=unpack)
    assert _whole(params, seen)


@pytest.mark.parametrize("spoil", [lambda t: t[:1], lambda t: t.double()])
def test_saved_come_back_as_something_else(library, spoil):
    with torch.autograd.graph.saved_tensors_hooks(lambda t: t, lambda t: spoil(t) if t.numel() == 8192 else t):
        _, _, _, (out, _) = _call()
    library.tsb_block_backward = None                     # (not reached)
    with pytest.raises(RuntimeError, match="came back"):
        out.backward(torch.zeros_like(out))
