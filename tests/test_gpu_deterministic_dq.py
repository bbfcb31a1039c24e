"""dQ of the deterministic backward: the exact sum of the fp32 contributions of its key tiles (64-bit fixed point), rounded once, so no
order of arrival and no other row changes its bits.  Bounds against the oracle as for the other tensor-core kernels (bf16 operands, dS
rounded to bf16): 2e-2 absolute, 5e-3 relative L2."""
import ctypes as C

import numpy as np
import pytest
import torch

from conftest import max_abs, rel_l2

pytestmark = pytest.mark.gpu
DETERMINISTIC = 4


@pytest.fixture(scope="module")
def sb():
    import sentinel_b200
    sentinel_b200._lib.load()
    assert torch.cuda.is_available()
    return sentinel_b200


def _inputs(B, Hq, Hkv, S, D, Skv=None):
    g = torch.Generator(device="cuda").manual_seed(S + D)
    make = lambda H, n, std: (torch.randn(B, H, n, D, generator=g, device="cuda") * std).to(torch.bfloat16)
    return make(Hq, S, 0.5), make(Hkv, Skv or S, 0.5), make(Hkv, Skv or S, 1.0), make(Hq, S, 1.0)


@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("B,Hq,Hkv,S,Skv,window,global_tokens,causal", [
    (1, 2, 1, 1, 1, 0, 0, True),
    (1, 2, 2, 128, 128, 0, 0, True),          # exactly one tile
    (2, 6, 2, 129, 129, 0, 0, True),          # one row and one key more
    (1, 4, 1, 1100, 1100, 0, 0, True),        # more tiles than stages
    (7, 24, 8, 200, 200, 0, 0, True),         # more blocks than SMs: blocks taken over
    (1, 2, 1, 700, 700, 130, 5, True),        # window edges inside tiles, global tokens
    (1, 2, 1, 900, 900, 64, 260, True),       # tiles skipped between the global tokens and the window
    (2, 4, 2, 150, 1000, 0, 0, False),        # rectangular, a ragged last key tile
])
def test_dq_against_the_oracle(sb, oracle, B, Hq, Hkv, S, Skv, window, global_tokens, causal, D):
    q, k, v, do = _inputs(B, Hq, Hkv, S, D, Skv)
    kw = dict(window=window, global_tokens=global_tokens, causal=causal)
    o, lse = sb.attention_forward(q, k, v, **kw)
    got = sb.attention_backward(q, k, v, o, lse, do, flags=DETERMINISTIC, **kw)
    assert sb.last_path() == "tcgen05" and sb.poll_device_status() == 0
    a = [t.float().cpu().numpy() for t in (q, k, v, do)]
    want = oracle.attn_bwd(*a, **kw)[:3]
    for x, w, name in zip(got, want, ("dq", "dk", "dv")):
        x = x.float().cpu().numpy()
        assert np.isfinite(x).all() and max_abs(x, w) <= 2e-2 * max(1.0, float(np.abs(w).max())), (name, max_abs(x, w))
        if float(np.abs(w).max()) > 1e-6:
            assert rel_l2(x, w) <= 5e-3, (name, rel_l2(x, w))
    # a part of the call gives the bits of the whole
    last = [t[B - 1:].contiguous() for t in (q, k, v, o, lse, do)]
    part = sb.attention_backward(*last, flags=DETERMINISTIC, **kw)
    assert torch.equal(part[0], got[0][B - 1:])


@pytest.mark.parametrize("flags", [0, DETERMINISTIC])
@pytest.mark.parametrize("D", [64, 128])
def test_gradients_in_the_place_of_the_operands(sb, D, flags):
    """dQ, dK and dV may lie where Q (or dO), K and V lie."""
    q, k, v, do = _inputs(2, 4, 4, 300, D)
    o, lse = sb.attention_forward(q, k, v)
    want = sb.attention_backward(q, k, v, o, lse, do, flags=flags)
    for outs in (lambda q, k, v, do: (q, k, v), lambda q, k, v, do: (do, k, v), lambda q, k, v, do: (torch.empty_like(q), k, v)):
        c = [t.clone() for t in (q, k, v, do)]
        dq, dk, dv = outs(*c)
        got = sb.attention_backward(*c[:3], o, lse, c[3], flags=flags, dq=dq, dk=dk, dv=dv)
        assert got[0].data_ptr() == dq.data_ptr()
        for x, w in zip(got, want):
            assert torch.equal(x, w) if flags or x is not got[0] else rel_l2(x.float().cpu().numpy(), w.float().cpu().numpy()) <= 1e-3


@pytest.mark.parametrize("D", [64, 128])
def test_dq_as_a_matrix_is_the_same(sb, D):
    """Feature-major fp32 matrices with bf16 operands allowed, against the token-major call on the rounded operands."""
    from sentinel_b200.flash_attention import CudaFlashAttention as F
    from sentinel_b200 import _lib
    B, H, S = 3, 4, 200
    q, k, v, do = _inputs(B, H, H, S, D)
    mats = [t.float().permute(1, 3, 0, 2).reshape(H * D, B * S).contiguous() for t in (q, k, v, do)]
    out = [torch.zeros(H * D, B * S, device="cuda") for _ in range(4)]
    lse = torch.zeros(H, B * S, device="cuda")
    shape = (H, D, D ** -0.5, True, 0, S, B)
    old = F.allow_reduced_precision
    F.allow_reduced_precision = True
    try:
        F.forwardMultiHead(*mats[:3], out[0], lse, *shape)
        d = F._desc(mats[0], mats[1], H, D, D ** -0.5, True, 0, S, B)
        d.flags |= _lib.FLAG_DETERMINISTIC
        import ctypes as C
        lib = _lib.load()
        ws = torch.empty(lib.sntl_attn_bwd_workspace_bytes(C.byref(d)), dtype=torch.uint8, device="cuda")
        rc = lib.sntl_attn_bwd(C.byref(d), *(t.data_ptr() for t in mats[:3]), out[0].data_ptr(), lse.data_ptr(), mats[3].data_ptr(),
                               *(t.data_ptr() for t in out[1:]), ws.data_ptr(), ws.numel(), torch.cuda.current_stream().cuda_stream)
    finally:
        F.allow_reduced_precision = old
    assert rc == 0 and sb.poll_device_status() == 0
    back = lambda m: m.reshape(H, D, B, S).permute(2, 0, 3, 1)
    o = back(out[0]).contiguous()
    ref = sb.attention_backward(q, k, v, o.to(torch.bfloat16), lse.reshape(H, B, S).permute(1, 0, 2).contiguous(), do, flags=DETERMINISTIC)
    # delta from O in fp32 there, from O rounded to bf16 here: as far apart as the rounding of O
    assert rel_l2(back(out[1]).cpu().numpy(), ref[0].float().cpu().numpy()) <= 5e-3


def _matrix_backward(sb, q, k, v, do, flags):
    """dQ of the feature-major call (fp32 matrices, bf16 operands allowed), as [B, H, S, D]: not rounded to bf16 at the end."""
    from sentinel_b200.flash_attention import CudaFlashAttention as F
    from sentinel_b200 import _lib
    B, H, S, D = q.shape
    mats = [t.float().permute(1, 3, 0, 2).reshape(H * D, B * S).contiguous() for t in (q, k, v, do)]
    out = [torch.zeros(H * D, B * S, device="cuda") for _ in range(4)]
    lse = torch.zeros(H, B * S, device="cuda")
    lib = _lib.load()
    d = F._desc(mats[0], mats[1], H, D, D ** -0.5, True, 0, S, B)
    d.flags |= flags | _lib.FLAG_ALLOW_BF16_COMPUTE
    size = max(lib.sntl_attn_fwd_workspace_bytes(C.byref(d)), lib.sntl_attn_bwd_workspace_bytes(C.byref(d)))
    ws = torch.empty(size, dtype=torch.uint8, device="cuda")
    stream = torch.cuda.current_stream().cuda_stream
    p = lambda *ts: [t.data_ptr() for t in ts]
    assert lib.sntl_attn_fwd(C.byref(d), *p(*mats[:3], out[0], lse, ws), size, stream) == 0
    assert lib.sntl_attn_bwd(C.byref(d), *p(*mats[:3], out[0], lse, mats[3], *out[1:], ws), size, stream) == 0
    assert sb.last_path() == "tcgen05_staged" and sb.poll_device_status() == 0
    return out[1].reshape(H, D, B, S).permute(2, 0, 3, 1)


@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("B,H,S,big", [(2, 3, 129, 1), (1, 2, 1000, 1), (3, 4, 200, 1), (2, 3, 300, 3e3)])
def test_dq_sums_the_contributions_of_the_call_without_the_flag(sb, B, H, S, big, D):
    """The two calls differ by the rounding of fp32 sums of up to 8 contributions: below 8 x 2^-24 of a row's largest partial sum.  (big: contributions beyond
    2^13 on both sides of the call's own.)"""
    q, k, v, do = _inputs(B, H, H, S, D)
    v, do = v * big, do * big
    plain, exact = (_matrix_backward(sb, q, k, v, do, f).cpu().numpy() for f in (0, DETERMINISTIC))
    assert rel_l2(exact, plain) <= 2e-6


@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("S,at,big", [(3 * 128, 2, 1), (3 * 128 + 40, 2, 1), (3 * 128, 2, 1024), (260 * 128 + 40, 258, 1), (260 * 128, 258, 1024)])
def test_large_contributions_that_cancel_leave_the_bits_of_the_others(sb, S, at, big, D):
    """The keys of tiles 0 and `at` agree in V and in the first half of their features, are of opposite sign and 2^10 times as large in the second, where Q
    is zero: their contributions to dQ there cancel exactly, and what the other keys give must come out as if they were zero there.  (More than 256
    tiles, and with `big` contributions beyond 2^13, are summed in another way on the way.)"""
    q, k, v, do = _inputs(1, 2, 2, 150, D, S)
    v, do = v * big, do * big
    h, a, b = D // 2, slice(0, 128), slice(at * 128, at * 128 + 128)
    q[..., h:] = 0
    k[:, :, b, :h] = k[:, :, a, :h]
    v[:, :, b] = v[:, :, a]
    k[:, :, b, h:] = -1024 * k[:, :, a, h:]
    k[:, :, a, h:] *= 1024
    zeros = k.clone()
    zeros[:, :, a, h:] = 0
    zeros[:, :, b, h:] = 0
    kw = dict(causal=False)
    o, lse = sb.attention_forward(q, k, v, **kw)
    got, want = (sb.attention_backward(q, x, v, o, lse, do, flags=DETERMINISTIC, **kw)[0] for x in (k, zeros))
    assert sb.poll_device_status() == 0
    assert float(want[..., h:].float().abs().max()) > 1e-4
    assert torch.equal(got, want)
