"""Exact fp32 through split products on the tensor cores (csrc/attn_f32_fwd_sm100.cu, attn_f32_bwd_sm100.cu): calls with enough work
and head_dim up to 64 take them by themselves, flags=FORCE_SIMT keeps the FMA kernels.

Bound against the fp64 oracle: a product of parts is within 2^-23 of its terms' size (the tensor core cuts off below 2^-24; the parts
left out are at most 2^-24 of a term, 2^-27 rms), the exponential and the sums of up to a few thousand such products add a few units
of 2^-24 of the result's size: 1e-6 relative L2 covers them (measured 1e-7 to 4e-7; the FMA kernels 1e-7 to 1.1e-6).
"""
import numpy as np
import pytest
import torch

from conftest import rel_l2

pytestmark = pytest.mark.gpu
FORCE_SIMT = 2
REL = 1e-6


@pytest.fixture(scope="module")
def sb():
    import sentinel_b200
    sentinel_b200._lib.load()
    assert torch.cuda.is_available()
    return sentinel_b200


def _inputs(seed, B, Hq, Hkv, S, D, Skv=None):
    g = torch.Generator(device="cuda").manual_seed(seed)
    Skv = Skv or S
    return [torch.randn(B, H, n, D, generator=g, device="cuda") for H, n in ((Hq, S), (Hkv, Skv), (Hkv, Skv), (Hq, S))]


def _launches(sb, f):
    n = sb.launch_count()
    r = f()
    return r, sb.launch_count() - n


def _both(sb, q, k, v, do, **kw):
    (o, lse), nf = _launches(sb, lambda: sb.attention_forward(q, k, v, **kw))
    g, nb = _launches(sb, lambda: sb.attention_backward(q, k, v, o, lse, do, **kw))
    assert sb.last_path() == "simt_f32" and sb.poll_device_status() == 0
    return (o, lse) + tuple(g), (nf, nb)


NAMES = ("o", "lse", "dq", "dk", "dv")


@pytest.mark.parametrize("B,Hq,Hkv,S,D,window,global_tokens,causal", [
    (8, 12, 12, 129, 64, 0, 0, True),       # a row more than a block, a KV tile with one token
    (4, 16, 16, 192, 64, 0, 0, True),       # half a block
    (2, 12, 4, 301, 62, 0, 0, True),        # ragged, head_dim not a multiple of 4, grouped heads
    (6, 24, 24, 128, 30, 0, 0, True),       # features filled up to 64; exactly one block
    (8, 40, 40, 191, 16, 0, 0, True),
    (2, 6, 2, 700, 64, 130, 5, True),       # window edges inside tiles, global tokens
    (3, 6, 6, 640, 64, 64, 130, True),      # global tokens beyond one tile of keys
    (2, 8, 4, 257, 64, 0, 0, False),
    (1, 12, 4, 1153, 48, 0, 0, True),       # many tiles
])
def test_against_the_oracle(sb, oracle, B, Hq, Hkv, S, D, window, global_tokens, causal):
    q, k, v, do = _inputs(S + D, B, Hq, Hkv, S, D)
    kw = dict(window=window, global_tokens=global_tokens, causal=causal)
    got, launches = _both(sb, q, k, v, do, **kw)
    assert launches == (2, 2)               # the tensor-core kernel and the FMA kernel for what it leaves
    a = [t.cpu().numpy() for t in (q, k, v, do)]
    want = oracle.attn_fwd(*a[:3], **kw) + tuple(oracle.attn_bwd(*a, **kw)[:3])
    for x, w, name in zip(got, want, NAMES):
        assert rel_l2(x.cpu().numpy(), w) <= REL, (name, rel_l2(x.cpu().numpy(), w))
    again, _ = _both(sb, q, k, v, do, **kw)
    assert all(torch.equal(x, y) for x, y in zip(got, again))


def test_keys_longer_than_queries(sb):
    """New tokens behind a fp32 cache, and a rectangular call without a causal mask."""
    q, k, v, do = _inputs(3, 2, 12, 6, 150, 64, 1000)
    o, n = _launches(sb, lambda: sb.attention_cached_forward(q, k, v, 900))
    o2, _ = sb.attention_cached_forward(q, k, v, 900, flags=FORCE_SIMT), 0
    assert n == 2 and all(rel_l2(x.cpu().numpy(), y.cpu().numpy()) <= REL for x, y in zip(o, o2))
    got, launches = _both(sb, q, k, v, do, causal=False)
    want, _ = _both(sb, q, k, v, do, causal=False, flags=FORCE_SIMT)
    assert launches == (2, 2)
    for x, w, name in zip(got, want, NAMES):
        assert rel_l2(x.cpu().numpy(), w.cpu().numpy()) <= 2 * REL, name


@pytest.mark.parametrize("offset", [0, 1, 3])
def test_matrices_and_unaligned_tensors(sb, offset):
    """Feature-major matrices with a column offset, and token-major tensors that start anywhere."""
    from sentinel_b200.flash_attention import CudaFlashAttention as F
    B, H, S, D = 4, 12, 160, 64
    q, k, v, do = _inputs(offset, B, H, H, S, D)
    want, _ = _both(sb, q, k, v, do)
    C = 5 + B * S + 2
    mats = []
    for t in (q, k, v, do):
        m = torch.full((H * D, C), float("nan"), device="cuda")
        m[:, 5:5 + B * S] = t.permute(1, 3, 0, 2).reshape(H * D, B * S)
        mats.append(m)
    out = {n: torch.zeros(H * D if n != "lse" else H, C, device="cuda") for n in NAMES}
    F.allow_reduced_precision = False
    shape = (H, D, D ** -0.5, True, 5, S, B)
    F.forwardMultiHead(*mats[:3], out["o"], out["lse"], *shape)
    F.backwardMultiHead(*mats[:3], out["o"], out["lse"], mats[3], out["dq"], out["dk"], out["dv"], None, *shape)
    for w, name in zip(want, NAMES):
        rows = 1 if name == "lse" else D
        x = out[name][:, 5:5 + B * S].reshape(H, rows, B, S).permute(2, 0, 3, 1).reshape(w.shape)
        assert torch.equal(x, w), name       # the same products in the same order
        assert not out[name][:, :5].any() and not out[name][:, 5 + B * S:].any()
    moved = []
    for t in (q, k, v, do):
        flat = torch.empty(t.numel() + offset, device="cuda")
        flat[offset:] = t.reshape(-1)
        moved.append(flat[offset:].view(t.shape))
    got, _ = _both(sb, *moved)
    assert all(torch.equal(x, y) for x, y in zip(got, want))


@pytest.mark.parametrize("window", [0, 40])
@pytest.mark.parametrize("bad", [float("nan"), float("inf"), -3.0e38, 2.0 ** 31, 1e-37])
def test_blocks_with_odd_values_are_the_fma_kernels(sb, bad, window):
    """A block that meets a value that its products do not take is computed by the FMA kernels, bit for bit; the others stay."""
    B, H, S, D = 2, 24, 300, 64
    q, k, v, do = _inputs(7, B, H, H, S, D)
    kw = dict(window=window)
    clean, _ = _both(sb, q, k, v, do, **kw)
    for t in (q, do, k, v):
        t[1, 3, 170::2, 5] = bad              # query and key tile 1 on of one head
    fma, _ = _both(sb, q, k, v, do, flags=FORCE_SIMT, **kw)
    o, lse = sb.attention_forward(q, k, v, **kw)
    # the backward of both from the same forward results
    got = (o, lse) + tuple(sb.attention_backward(q, k, v, fma[0], fma[1], do, **kw))
    want = fma[:2] + tuple(sb.attention_backward(q, k, v, fma[0], fma[1], do, flags=FORCE_SIMT, **kw))
    assert sb.poll_device_status() == 0
    same = lambda x, y: torch.equal(x.nan_to_num(7.0), y.nan_to_num(7.0)) and torch.equal(x.isnan(), y.isnan())
    for x, w, c, name in zip(got, want, clean, NAMES):
        assert same(x[1, 3, 128:], w[1, 3, 128:]), name
        if name in ("o", "lse"):
            assert torch.equal(x[1, 3, :128], c[1, 3, :128]), name      # sees no such token
        if name in ("o", "lse"):
            assert torch.equal(x[0], c[0]) and torch.equal(x[1, :3], c[1, :3]) and torch.equal(x[1, 4:], c[1, 4:]), name


@pytest.mark.parametrize("bad", [float("nan"), 2.0 ** 31])
@pytest.mark.parametrize("Hq,Hkv,S,D", [(24, 24, 300, 64), (24, 8, 300, 48), (24, 8, 420, 30)])
def test_odd_blocks_and_no_others_are_left_to_the_fma_kernels(sb, Hq, Hkv, S, D, bad):
    """Values that the products do not take in one query head and its KV head: the blocks that meet them have the FMA kernels' bits, all others, of
    every result, those of the call without such values (and with the same O and LSE)."""
    B, group = 2, Hq // Hkv
    hq = 4
    hk, heads = hq // group, slice(hq // group * group, hq // group * group + group)
    clean = _inputs(7, B, Hq, Hkv, S, D)
    odd = [t.clone() for t in clean]
    for t, h in zip(odd, (hq, hk, hk, hq)):
        t[1, h, 170::2, 5] = bad              # tokens of row tile 1 on
    (o, lse), n = _launches(sb, lambda: sb.attention_forward(*odd[:3]))
    fo, flse = sb.attention_forward(*odd[:3], flags=FORCE_SIMT)
    co, clse = sb.attention_forward(*clean[:3])
    assert n == 2
    got, n = _launches(sb, lambda: sb.attention_backward(*odd[:3], fo, flse, odd[3]))
    fma = sb.attention_backward(*odd[:3], fo, flse, odd[3], flags=FORCE_SIMT)
    same_o = sb.attention_backward(*clean[:3], fo, flse, clean[3])
    assert n == 2 and sb.poll_device_status() == 0
    same = lambda x, y: torch.equal(x.nan_to_num(7.0), y.nan_to_num(7.0)) and torch.equal(x.isnan(), y.isnan())
    for x, f, c, per_query in ((o, fo, co, True), (lse, flse, clse, True), (got[0], fma[0], same_o[0], True), (got[1], fma[1], same_o[1], False),
                               (got[2], fma[2], same_o[2], False)):
        mine = heads if per_query else slice(hk, hk + 1)
        first = 128 if per_query else 0       # query tile 0 sees no such token; every key tile is seen by some
        assert same(x[1, mine, first:], f[1, mine, first:])
        others = torch.ones(x.shape[:3], dtype=torch.bool, device="cuda")
        others[1, mine, first:] = False
        # (O and LSE of the odd rows enter the backward of the clean call, but other heads' and rows' blocks do not read them)
        assert torch.equal(x[others], c[others])


@pytest.mark.parametrize("D,S", [(62, 333), (48, 333), (30, 500)])
@pytest.mark.parametrize("bad", [None, float("inf")])
def test_matrices_with_grouped_heads(sb, D, S, bad):
    """Feature-major matrices, grouped heads, head_dims that are not multiples of 8: the bits of the token-major call."""
    from sentinel_b200.flash_attention import CudaFlashAttention as F
    B, Hq, Hkv = 3, 12, 4
    q, k, v, do = _inputs(41, B, Hq, Hkv, S, D)
    if bad is not None:
        for t in (q, k, v, do):
            t[2, 1, 200, 3] = bad
    want, launches = _both(sb, q, k, v, do)
    assert launches == (2, 2)
    C = 3 + B * S + 6
    mats = []
    for t in (q, k, v, do):
        m = torch.full((t.shape[1] * D, C), 5.0, device="cuda")
        m[:, 3:3 + B * S] = t.permute(1, 3, 0, 2).reshape(-1, B * S)
        mats.append(m)
    out = {n: torch.zeros({"o": Hq * D, "dq": Hq * D, "lse": Hq}.get(n, Hkv * D), C, device="cuda") for n in NAMES}
    F.allow_reduced_precision = False
    shape = (Hq, D, D ** -0.5, True, 3, S, B)
    F.forwardMultiHead(*mats[:3], out["o"], out["lse"], *shape)
    F.backwardMultiHead(*mats[:3], out["o"], out["lse"], mats[3], out["dq"], out["dk"], out["dv"], None, *shape)
    assert sb.poll_device_status() == 0
    for w, name in zip(want, NAMES):
        x = out[name][:, 3:3 + B * S].reshape(w.shape[1], -1, B, S).permute(2, 0, 3, 1).reshape(w.shape)
        assert torch.equal(x.nan_to_num(7.0), w.nan_to_num(7.0)) and torch.equal(x.isnan(), w.isnan()), name


@pytest.mark.parametrize("scale", [2.0 ** -16, 3e-4, 3.0, 2.0 ** 16])
def test_scales(sb, scale):
    """Against the FMA kernels.  Scaled scores reach 150 for the scales above 1 and are known to a few 2^-24 of that, which is the error of a weight."""
    q, k, v, do = _inputs(43, 2, 24, 24, 300, 48)
    q = q / max(1.0, scale * 0.2)
    got, launches = _both(sb, q, k, v, do, scale=scale)
    want, _ = _both(sb, q, k, v, do, scale=scale, flags=FORCE_SIMT)
    assert launches == (2, 2)
    for x, w in zip(got, want):
        assert rel_l2(x.cpu().numpy(), w.cpu().numpy()) <= 4e-5


def test_streams_and_graphs(sb):
    """Two streams at once and a captured call give the bits of calls one by one."""
    sets = [_inputs(seed, 2, 24, 24, 300, 64) for seed in (47, 48)]
    want = [_both(sb, *x)[0] for x in sets]
    streams = [torch.cuda.Stream() for _ in sets]
    got = [[] for _ in sets]
    torch.cuda.synchronize()
    for _ in range(8):
        for st, x, r in zip(streams, sets, got):
            with torch.cuda.stream(st):
                o, lse = sb.attention_forward(*x[:3])
                r.append((o, lse) + tuple(sb.attention_backward(*x[:3], o, lse, x[3])))
    torch.cuda.synchronize()
    assert all(torch.equal(a, b) for w, rs in zip(want, got) for r in rs for a, b in zip(r, w))
    x = [t.clone() for t in sets[0]]
    st = torch.cuda.Stream()
    with torch.cuda.stream(st):
        _both(sb, *x)
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g, stream=st):
            o, lse = sb.attention_forward(*x[:3])
            r = (o, lse) + tuple(sb.attention_backward(*x[:3], o, lse, x[3]))
    for inputs, w in zip(sets, want):
        for t, y in zip(x, inputs):
            t.copy_(y)
        torch.cuda.synchronize()
        g.replay()
        torch.cuda.synchronize()
        assert all(torch.equal(a, b) for a, b in zip(r, w))


def test_inconsistent_lse_is_the_fma_kernels(sb):
    """Weights far above 1 (an LSE that is not this call's) would overflow in parts: the FMA kernels' results, infinities included."""
    q, k, v, do = _inputs(11, 2, 24, 24, 256, 64)
    o, lse = sb.attention_forward(q, k, v)
    lse[0, 1, 200] = -120.0
    lse[1, 0, 3] = float("nan")
    lse[1, 1, 4] = float("inf")
    got = sb.attention_backward(q, k, v, o, lse, do)
    want = sb.attention_backward(q, k, v, o, lse, do, flags=FORCE_SIMT)
    for x, w in zip(got, want):
        assert torch.equal(x.isfinite(), w.isfinite())
        fin = w.isfinite()
        assert float((x - w)[fin].norm() / w[fin].norm()) <= 2 * REL


@pytest.mark.parametrize("Hq,Hkv,T,L,D,window,launches", [
    (4, 4, 64, 8192, 64, 0, 1),       # 64 tiles of 128 keys in one chain on four SMs (200 us; the FMA kernels over clusters: 85)
    (1, 1, 1024, 1024, 64, 0, 1),     # 33 / 22
    (2, 1, 154, 1996, 64, 0, 1),      # 57 / 25
    (12, 12, 256, 2048, 64, 0, 2),    # 57 / 100
    (4, 4, 512, 2048, 64, 0, 2),      # 57 / 82
    (12, 12, 1024, 1024, 32, 16, 1),  # hidden pairs are no work: 15.6 / 14.4
    (12, 12, 1024, 1024, 32, 256, 2), # 19 / 29
])
def test_route_follows_the_chains_and_the_mask(sb, Hq, Hkv, T, L, D, window, launches):
    """The tensor-core kernel (a second launch looks for its marks) takes a call where its chains of tiles are shorter than the FMA kernels'."""
    q, k, v, _ = _inputs(19, 1, Hq, Hkv, T, D, L)
    (o, lse), n = _launches(sb, lambda: sb.attention_cached_forward(q, k, v, L, window=window))
    assert n == launches and sb.last_path() == "simt_f32" and sb.poll_device_status() == 0
    for x, y in zip((o, lse), sb.attention_cached_forward(q, k, v, L, window=window, flags=FORCE_SIMT)):
        assert rel_l2(x.cpu().numpy(), y.cpu().numpy()) <= REL


@pytest.mark.parametrize("exponent", [10, 16, 24, 31, 40])
@pytest.mark.parametrize("D", [32, 48, 64])
def test_large_scores_of_rows_with_one_key(sb, D, exponent):
    """Scores around 2^exponent, each row's own far above its others: the weight is 1, not exp of the rounding error of its scaled score (half a unit
    in the last place of the score; at D 32 and 48, whose scale is no power of two).  O is V and the LSE the score."""
    B, H, S = 2, 24, 256
    _, _, v, _ = _inputs(17, B, H, H, S, D)
    g = torch.Generator(device="cuda").manual_seed(18)
    rand = lambda *shape: torch.rand(*shape, generator=g, device="cuda")
    k = torch.where(rand(B, H, S, D) < 0.5, -1.0, 1.0) * (0.9 + 0.2 * rand(B, H, 1, D)) * 2.0 ** (exponent / 2)
    q = k * (1 + rand(B, H, S, 1)) * D ** -0.5
    x = torch.einsum("bhqd,bhkd->bhqk", q.double(), k.double()) * float(np.float32(D ** -0.5))
    own = x.diagonal(dim1=-2, dim2=-1)
    assert float((own - x.masked_fill(torch.eye(S, device="cuda").bool(), -float("inf")).amax(-1)).min()) > 20
    (o, lse), launches = _launches(sb, lambda: sb.attention_forward(q, k, v))
    assert launches == 2 and sb.poll_device_status() == 0
    for x, w in ((o, v), (lse, own)):
        assert rel_l2(x.cpu().numpy(), w.cpu().numpy()) <= REL


def _exact(q, k, v, do):
    q, k, v, do = (t.double() for t in (q, k, v, do))
    scale = float(np.float32(q.shape[-1] ** -0.5))
    p = torch.softmax(q @ k.transpose(-1, -2) * scale, -1)
    o = p @ v
    ds = p * (do @ v.transpose(-1, -2) - (do * o).sum(-1, keepdim=True)) * scale
    return p, o, ds @ k, ds.transpose(-1, -2) @ q, p.transpose(-1, -2) @ do


@pytest.mark.parametrize("D", [48, 64])
def test_weights_near_the_smallest(sb, D):
    """A token that every row gives a weight of about 2^-124, whose V is all that is not zero in some features: the parts of such weights have no room
    in bf16.  Bound: scores of size 86 are known to 2^-23 of it, so their exponentials to 1e-5."""
    q, k, v, do = _inputs(23, 1, 24, 24, 300, D)
    q[..., 0], k[..., 0] = 8.0, 0.0
    k[:, :, 0] = 0.0
    k[:, :, 0, 0] = -80.0 / 8 * D ** 0.5
    v[:, :, 1:, :5] = 0.0
    got, launches = _both(sb, q, k, v, do, causal=False)
    assert launches == (2, 2)
    p, o, dq, dk, dv = _exact(q, k, v, do)
    assert 2.0 ** -126 < float(p[..., 0].min()) and float(p[..., 0].max()) < 2.0 ** -112
    for x, w in ((got[0][..., :5], o[..., :5]), (got[4][:, :, 0], dv[:, :, 0]), (got[3][:, :, 0], dk[:, :, 0])):
        assert rel_l2(x.double().cpu().numpy() * 2.0 ** 120, w.cpu().numpy() * 2.0 ** 120) <= 1e-5


@pytest.mark.parametrize("D", [48, 64])
def test_gradients_near_the_smallest(sb, D):
    """dO around 2^-114, of so few bits that its parts add up to it: dS around 2^-122 and below has to keep its bits."""
    q, k, v, do = _inputs(29, 1, 24, 24, 300, D)
    do = (do.sign() * do.abs().clamp(0.25, 4.0)).to(torch.bfloat16).float() * 2.0 ** -114
    got, launches = _both(sb, q, k, v, do, causal=False)
    assert launches == (2, 2)
    for x, w in zip(got[2:], _exact(q, k, v, do)[2:]):
        assert rel_l2(x.double().cpu().numpy() * 2.0 ** 110, w.cpu().numpy() * 2.0 ** 110) <= 2 * REL


@pytest.mark.parametrize("flags", [4, 16])       # SNTL_FLAG_DETERMINISTIC, SNTL_FLAG_WHOLE_KEY_TILES
@pytest.mark.parametrize("B,Hq,Hkv,S,D,window", [(8, 4, 4, 256, 64, 0), (8, 6, 2, 100, 64, 0), (8, 4, 2, 300, 32, 0), (8, 8, 8, 640, 16, 70)])
def test_gradients_of_a_part_have_the_bits_of_the_whole(sb, flags, B, Hq, Hkv, S, D, window):
    q, k, v, do = _inputs(31, B, Hq, Hkv, S, D)
    o, lse = sb.attention_forward(q, k, v, window=window)
    kw = dict(flags=flags, window=window)
    whole, n = _launches(sb, lambda: sb.attention_backward(q, k, v, o, lse, do, **kw))
    assert n == (2 if S * D >= 8192 else 1)
    for b, h in ((3, slice(0, Hkv)), (5, slice(Hkv - 1, Hkv))):
        g = slice(h.start * Hq // Hkv, h.stop * Hq // Hkv)
        part = [t[b:b + 1, g].contiguous() for t in (q, o, lse, do)]
        kv = [t[b:b + 1, h].contiguous() for t in (k, v)]
        got = sb.attention_backward(part[0], *kv, *part[1:], **kw)
        assert all(torch.equal(x, y[b:b + 1, s]) for x, y, s in zip(got, whole, (g, h, h)))


@pytest.mark.parametrize("B,H,S,D", [(8, 16, 224, 64), (4, 4, 256, 64), (2, 4, 300, 96)])
def test_deterministic_host_pipeline_has_the_bits_of_one_call(sb, B, H, S, D):
    from sentinel_b200.host_pipeline import forward_backward_host
    q, k, v, do = _inputs(37, B, H, H, S, D)
    o, lse = sb.attention_forward(q, k, v, flags=4)
    want = (o, lse) + tuple(sb.attention_backward(q, k, v, o, lse, do, flags=4))
    got = forward_backward_host(*(t.cpu().pin_memory() for t in (q, k, v, do)), flags=4)
    assert all(torch.equal(x, y.cpu()) for x, y in zip(got, want))
