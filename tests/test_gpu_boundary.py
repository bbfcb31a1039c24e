"""GPU tests of the boundary contract: the host-buffer call (transfers overlapped with the kernels) returns the same
results as the device-resident calls, and the C-ABI calls can be captured into a CUDA graph and replayed, which is how
the reference's trainer drives its attention (CudaLanguageModel.cu:2176-2209: two eager warm-ups, then capture/replay)."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def sb():
    import sentinel_b200
    sentinel_b200._lib.load()
    return sentinel_b200


def test_host_buffer_call_matches_device_calls(sb):
    w = sb.WORKLOADS["gqa7b_d128"]
    q, k, v, do = (t.pin_memory() for t in sb.make_inputs(w, batch=3, q_heads=4, kv_heads=2, seq=640))
    qd, kd, vd, dod = (t.cuda() for t in (q, k, v, do))
    o, lse = sb.attention_forward(qd, kd, vd)
    dq, dk, dv = sb.attention_backward(qd, kd, vd, o, lse, dod)
    for chunks in (None, 1, 2, 6):      # KV-group chunks, whole problem, batch chunks, one chunk per unit
        from sentinel_b200.host_pipeline import forward_backward_host
        ho, hl, hdq, hdk, hdv = forward_backward_host(q, k, v, do, chunks=chunks)
        assert torch.equal(ho, o.cpu()) and torch.equal(hl, lse.cpu())
        assert torch.equal(hdk, dk.cpu()) and torch.equal(hdv, dv.cpu())          # one owner each: bit-identical
        assert float((hdq.float() - dq.cpu().float()).abs().max()) <= 1e-3 * float(dq.float().abs().max())  # reduction order varies
    assert sb.poll_device_status() == 0


def test_c_abi_calls_are_graph_capturable(sb):
    w = sb.WORKLOADS["gqa7b_d128"]
    q, k, v, do = (t.cuda() for t in sb.make_inputs(w, batch=1, q_heads=4, kv_heads=1, seq=512))
    o, lse = torch.empty_like(q), torch.empty(q.shape[:3], dtype=torch.float32, device="cuda")
    dq, dk, dv = torch.empty_like(q), torch.empty_like(k), torch.empty_like(v)

    def step():
        sb.attention_forward(q, k, v, out=o, lse=lse)
        sb.attention_backward(q, k, v, o, lse, do, dq=dq, dk=dk, dv=dv)

    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        for _ in range(2):               # eager warm-ups: kernel attributes set, scratch grown
            step()
    torch.cuda.current_stream().wait_stream(side)
    torch.cuda.synchronize()
    want = [t.clone() for t in (o, lse, dk, dv)]
    want_dq = dq.clone()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        step()
    for t in (o, lse, dq, dk, dv):
        t.zero_()
    graph.replay()
    graph.replay()
    torch.cuda.synchronize()
    for got, ref in zip((o, lse, dk, dv), want):
        assert torch.equal(got, ref)
    assert float((dq.float() - want_dq.float()).abs().max()) <= 1e-3 * float(want_dq.float().abs().max())
    assert sb.poll_device_status() == 0


def test_calls_on_two_streams_keep_their_scratch_apart(sb):
    """Backward calls that overlap on the GPU (two streams, as in the host-buffer pipeline's two compute streams) must
    not share scratch: each stream's results equal those of the same call run alone."""
    w = sb.WORKLOADS["gqa7b_d128"]
    cases = []
    for seed in (0, 1):
        q, k, v, do = (t.cuda() for t in sb.make_inputs(w, batch=1, q_heads=7, kv_heads=1, seq=1024, seed_offset=seed))
        o, lse = sb.attention_forward(q, k, v)
        dq, dk, dv = sb.attention_backward(q, k, v, o, lse, do)
        cases.append((q, k, v, do, o, lse, dq.clone(), dk.clone(), dv.clone()))
    torch.cuda.synchronize()
    streams = [torch.cuda.Stream(), torch.cuda.Stream()]
    for _ in range(5):
        outs = []
        for st, (q, k, v, do, o, lse, *_ref) in zip(streams, cases):
            st.wait_stream(torch.cuda.current_stream())
            with torch.cuda.stream(st):
                outs.append(sb.attention_backward(q, k, v, o, lse, do))
        torch.cuda.synchronize()
        for (dq, dk, dv), case in zip(outs, cases):
            assert torch.equal(dk, case[7]) and torch.equal(dv, case[8])
            assert float((dq.float() - case[6].float()).abs().max()) <= 1e-3 * float(case[6].float().abs().max())
    assert sb.poll_device_status() == 0


def test_bounded_wait_runs_out_reports_and_leaves_the_context_usable(sb):
    """Failure detection without a fault: a small kernel waits, with a 2 ms limit, on barriers that by construction
    never receive their arrival.  The waits run out as a stuck production wait would after its one second: the
    kernel returns normally, the poll reports SNTL_ERR_DEVICE_TIMEOUT with the self-test's site code, the report is
    cleared by that poll, and the next real call (made after the short give-up window has passed) is clean and exact."""
    import ctypes as C
    import time
    from sentinel_b200 import _lib
    lib = _lib.load()
    assert sb.poll_device_status() == 0
    stream = torch.cuda.current_stream().cuda_stream
    assert lib.sntl_attn_selftest_wait_timeout(2000, stream) == _lib.OK
    fwd, bwd = C.c_uint32(0), C.c_uint32(0)
    rc = lib.sntl_attn_poll_device_status_words(stream, C.byref(fwd), C.byref(bwd))
    assert rc == _lib.ERR_DEVICE_TIMEOUT
    assert fwd.value >> 24 == 0x7e and bwd.value == 0
    assert lib.sntl_attn_poll_device_status_words(stream, C.byref(fwd), C.byref(bwd)) == _lib.OK   # cleared by the poll
    with pytest.raises(RuntimeError):      # the python mirror raises at its synchronisation point
        assert lib.sntl_attn_selftest_wait_timeout(1000, stream) == _lib.OK
        sb.raise_if_device_wait_timed_out()
    time.sleep(0.05)                       # well past the 1-2 ms during which other waits would give up early
    w = sb.WORKLOADS["gqa7b_d128"]
    q, k, v, do = (t.cuda() for t in sb.make_inputs(w, batch=1, q_heads=4, kv_heads=2, seq=512))
    o1, lse1 = sb.attention_forward(q, k, v)
    dq1, dk1, dv1 = sb.attention_backward(q, k, v, o1, lse1, do)
    assert sb.poll_device_status() == 0
    o2, lse2 = sb.attention_forward(q, k, v)
    assert torch.equal(o1, o2) and torch.equal(lse1, lse2)
    assert lib.sntl_attn_selftest_wait_timeout(0, stream) == _lib.ERR_BAD_ARGUMENT
    assert lib.sntl_attn_selftest_wait_timeout(200000, stream) == _lib.ERR_BAD_ARGUMENT


@pytest.mark.parametrize("limit_us", [1, 2000, 50000])
def test_every_form_of_bounded_wait_runs_out(sb, limit_us):
    """The wait of one thread, its short form in a thread and in a warp, and warps that meet in a named barrier after some of them have
    given up: each returns false, sets the flag of its block and, when nothing else has given up, takes its limit, not the kernels' one
    second (the self-test records site 0x7d instead of 0x7e if one does not).  The next call after it is clean."""
    import ctypes as C
    import time
    from sentinel_b200 import _lib
    lib = _lib.load()
    assert sb.poll_device_status() == 0
    time.sleep(0.12)                       # (past what an earlier self-test makes other waits give up early)
    stream = torch.cuda.current_stream().cuda_stream
    torch.cuda.synchronize()
    t0 = time.perf_counter()
    assert lib.sntl_attn_selftest_wait_timeout(limit_us, stream) == _lib.OK
    torch.cuda.synchronize()
    assert limit_us * 1e-6 <= time.perf_counter() - t0 < 0.5 + limit_us * 1e-6
    fwd, bwd = C.c_uint32(0), C.c_uint32(0)
    assert lib.sntl_attn_poll_device_status_words(stream, C.byref(fwd), C.byref(bwd)) == _lib.ERR_DEVICE_TIMEOUT
    assert fwd.value >> 24 == 0x7e and fwd.value & 0xffffff < 4 and bwd.value == 0
    time.sleep(0.12)
    q = torch.randn(1, 2, 300, 64, device="cuda", dtype=torch.bfloat16)
    o, _ = sb.attention_forward(q, q, q)
    assert sb.poll_device_status() == 0 and bool(torch.isfinite(o).all())


def test_deterministic_flag_makes_dq_bit_reproducible(sb):
    """SNTL_FLAG_DETERMINISTIC: dQ is summed in 64-bit fixed point, so it is bit-identical from run to run, between the
    one-stream and two-stream variants and through the chunked host-buffer pipeline -- and it meets the same oracle
    bounds as the default path (it is the exact sum of the same fp32 contributions, rounded once)."""
    import numpy as np
    from oracle import cpu
    from sentinel_b200 import _lib
    from sentinel_b200.host_pipeline import forward_backward_host
    det = _lib.FLAG_DETERMINISTIC
    for name, kw in (("gqa7b_d128", dict(batch=2, q_heads=8, kv_heads=2, seq=1152)), ("llama1b_gqa", dict(batch=1, q_heads=8, kv_heads=4, seq=777))):
        w = sb.WORKLOADS[name]
        q, k, v, do = (t.pin_memory() for t in sb.make_inputs(w, **kw))
        qd, kd, vd, dod = (t.cuda() for t in (q, k, v, do))
        o, lse = sb.attention_forward(qd, kd, vd)
        dq1, dk1, dv1 = sb.attention_backward(qd, kd, vd, o, lse, dod, flags=det)
        runs = [sb.attention_backward(qd, kd, vd, o, lse, dod, flags=det) for _ in range(4)]
        side = torch.cuda.Stream()
        side.wait_stream(torch.cuda.current_stream())
        with torch.cuda.stream(side):
            runs.append(sb.attention_backward(qd, kd, vd, o, lse, dod, flags=det))
        runs.append(sb.attention_backward(qd, kd, vd, o, lse, dod, flags=det))     # overlaps the side stream's call
        torch.cuda.synchronize()
        for dq, dk, dv in runs:
            assert torch.equal(dq, dq1) and torch.equal(dk, dk1) and torch.equal(dv, dv1)
        for chunks in (None, 1, 2):
            _, _, hdq, hdk, hdv = forward_backward_host(q, k, v, do, chunks=chunks, flags=det)
            assert torch.equal(hdq, dq1.cpu()) and torch.equal(hdk, dk1.cpu()) and torch.equal(hdv, dv1.cpu())
        # the default path differs from it only in the last bits, and both sit inside the oracle bounds
        dq0, _, _ = sb.attention_backward(qd, kd, vd, o, lse, dod)
        assert float((dq0.float() - dq1.float()).abs().max()) <= 1e-2 * float(dq1.float().abs().max())
        wdq, wdk, wdv, _ = cpu.attn_bwd(*(t.float().numpy() for t in (q, k, v, do)))
        got = dq1.float().cpu().numpy()
        assert float(np.abs(got - wdq).max()) <= 2e-2
        assert float(np.linalg.norm(got - wdq) / np.linalg.norm(wdq)) <= 5e-3
    assert sb.poll_device_status() == 0


def _offset(t, elements):
    """The same values in a contiguous tensor that starts `elements` elements past an allocation."""
    x = torch.empty(t.numel() + elements, dtype=t.dtype, device=t.device)[elements:].view(t.shape)
    return x.copy_(t)


@pytest.mark.parametrize("D", [64, 128])
def test_backward_reads_o_from_any_8_byte_boundary(sb, D):
    """O has no tensor map and is read by the pre-pass alone: a view 8 bytes past a 16-byte boundary gives the same bits."""
    g = torch.Generator(device="cuda").manual_seed(D)
    q, do = (torch.randn(2, 4, 201, D, generator=g, device="cuda").to(torch.bfloat16) for _ in range(2))
    k, v = (torch.randn(2, 2, 201, D, generator=g, device="cuda").to(torch.bfloat16) for _ in range(2))
    o, lse = sb.attention_forward(q, k, v)
    want = sb.attention_backward(q, k, v, o, lse, do, flags=4)
    view = _offset(o, 4)
    assert view.data_ptr() % 16 == 8
    for got, ref in zip(sb.attention_backward(q, k, v, view, lse, do, flags=4), want):
        assert torch.equal(got, ref)
    # the backward in pieces reads dO that way too, before any product needs its tensor map
    dk, dv = torch.zeros(k.shape, device="cuda"), torch.zeros(v.shape, device="cuda")
    pieces = sb.BackwardPieces(q, view, lse, do)
    pieces.block(k, v, dk, dv, causal=True)
    assert float((pieces.end().float() - want[0].float()).norm() / want[0].float().norm()) <= 4e-3   # bf16 rounding of both
    assert sb.poll_device_status() == 0


def test_misaligned_tensors_are_refused_before_any_launch(sb):
    """The tensor-core kernels access bf16 tensors and scratch 16 bytes at a time (O 8): other addresses are an error, and
    nothing is launched.  (Only the refusal is tested: no kernel runs on such an address.)"""
    import ctypes as C
    from sentinel_b200 import _lib
    lib = _lib.load()
    g = torch.Generator(device="cuda").manual_seed(1)
    q, do = (torch.randn(1, 4, 256, 64, generator=g, device="cuda").to(torch.bfloat16) for _ in range(2))
    k, v = (torch.randn(1, 2, 256, 64, generator=g, device="cuda").to(torch.bfloat16) for _ in range(2))
    o, lse = sb.attention_forward(q, k, v)
    sb.attention_backward(q, k, v, o, lse, do)
    before = sb.launch_count()
    args = dict(q=q, k=k, v=v, o=o, lse=lse, dout=do, dq=torch.empty_like(q), dk=torch.empty_like(k), dv=torch.empty_like(v))
    for name in ("q", "k", "v", "dout", "dq", "dk", "dv", "o"):
        with pytest.raises(RuntimeError):
            sb.attention_backward(**{**args, name: _offset(args[name], 1 if name == "o" else 4)})
    for name in ("q", "k", "v", "out"):
        with pytest.raises(RuntimeError):
            sb.attention_forward(**{**dict(q=q, k=k, v=v, out=torch.empty_like(q)), name: _offset(q if name in ("q", "out") else k, 4)})
    with pytest.raises(RuntimeError):
        sb.BackwardPieces(q, _offset(o, 1), lse, do)
    with pytest.raises(RuntimeError):
        sb.BackwardPieces(q, o, lse, _offset(do, 2))
    # scratch, of the direct and of the staged calls
    stream = torch.cuda.current_stream().cuda_stream
    scratch = torch.empty(1 << 24, dtype=torch.uint8, device="cuda")
    for dtype, layout, flags in ((_lib.DTYPE_BF16, _lib.LAYOUT_BHSD, 0), (_lib.DTYPE_F32, _lib.LAYOUT_SENTINEL, _lib.FLAG_ALLOW_BF16_COMPUTE)):
        d = _lib.Desc(dtype, layout, 1, 4, 2, 256, 256, 64, 0.125, 1, 256, 0, flags)
        m = [torch.empty(256 * 256 * 4, device="cuda") for _ in range(9)]
        p = [t.data_ptr() for t in m]
        assert lib.sntl_attn_bwd(C.byref(d), *p, scratch.data_ptr() + 8, 1 << 23, stream) == _lib.ERR_CUDA
        if layout == _lib.LAYOUT_SENTINEL:
            assert lib.sntl_attn_fwd(C.byref(d), *p[:5], scratch.data_ptr() + 8, 1 << 23, stream) == _lib.ERR_CUDA
    assert sb.launch_count() == before
    torch.cuda.synchronize()                 # no error is pending


def test_out_of_memory_for_scratch_is_torchs_own_error(sb):
    """A call whose scratch cannot be allocated raises torch.OutOfMemoryError (what retry and batch-shrinking code catches), and
    the same call works once there is memory.  The process's own limit is lowered; the GPU's memory is not exhausted."""
    g = torch.Generator(device="cuda").manual_seed(5)
    q, do = (torch.randn(2, 16, 8192, 128, generator=g, device="cuda").to(torch.bfloat16) for _ in range(2))
    k, v = (torch.randn(2, 4, 8192, 128, generator=g, device="cuda").to(torch.bfloat16) for _ in range(2))
    o, lse = sb.attention_forward(q, k, v)
    out = dict(dq=torch.empty_like(q), dk=torch.empty_like(k), dv=torch.empty_like(v))
    stream = torch.cuda.Stream()
    stream.wait_stream(torch.cuda.current_stream())
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    total = torch.cuda.get_device_properties(0).total_memory
    torch.cuda.set_per_process_memory_fraction((torch.cuda.memory_reserved() + (64 << 20)) / total)
    try:
        with torch.cuda.stream(stream), pytest.raises(torch.OutOfMemoryError):
            sb.attention_backward(q, k, v, o, lse, do, flags=4, **out)      # 270 MB of 64-bit dQ words and more
    finally:
        torch.cuda.set_per_process_memory_fraction(1.0)
    with torch.cuda.stream(stream):
        sb.attention_backward(q, k, v, o, lse, do, flags=4, **out)
    torch.cuda.synchronize()
    assert sb.poll_device_status() == 0 and bool(torch.isfinite(out["dq"]).all())


def test_threads_on_one_stream_keep_their_scratch_apart(sb):
    """Python threads share the default stream, and the interpreter lock is given up while a call launches its kernels: the kernels
    of two calls must not alternate on one buffer.  Different problems in each thread, every result as when called alone."""
    import sys
    import threading
    cases = []
    for seed, (H, S, D) in enumerate(((8, 384, 64), (3, 640, 128), (12, 200, 64))):
        g = torch.Generator(device="cuda").manual_seed(seed)
        q, do, k, v = (torch.randn(1, H, S, D, generator=g, device="cuda").to(torch.bfloat16) for _ in range(4))
        o, lse = sb.attention_forward(q, k, v)
        cases.append(((q, k, v, o, lse, do), [t.clone() for t in sb.attention_backward(q, k, v, o, lse, do, flags=4)]))
    torch.cuda.synchronize()
    wrong = []

    def work(args, want):
        for _ in range(150):
            got = sb.attention_backward(*args, flags=4)
            if not all(torch.equal(x, y) for x, y in zip(got, want)):
                wrong.append(args[0].shape)

    switch = sys.getswitchinterval()
    sys.setswitchinterval(1e-5)
    try:
        threads = [threading.Thread(target=work, args=c) for c in cases for _ in range(2)]
        for t in threads:
            t.start()
        for t in threads:
            t.join()
    finally:
        sys.setswitchinterval(switch)
    assert not wrong and sb.poll_device_status() == 0


@pytest.mark.parametrize("warm", [True, False])
def test_scratch_of_a_captured_call_stays_with_its_graph(sb, warm):
    """A call is captured on a stream that has made the same call before, or has not; a larger call then replaces that stream's
    scratch, and other tensors take its place.  A replay gives the same results and leaves those tensors alone."""
    g = torch.Generator(device="cuda").manual_seed(9)
    q, do, k, v = (torch.randn(1, 4, 512, 64, generator=g, device="cuda").to(torch.bfloat16) for _ in range(4))
    big = [torch.randn(2, 8, 2048, 64, generator=g, device="cuda").to(torch.bfloat16) for _ in range(4)]
    o, lse = sb.attention_forward(q, k, v)
    big_o, big_lse = sb.attention_forward(*big[:3])
    grads = dict(dq=torch.empty_like(q), dk=torch.empty_like(k), dv=torch.empty_like(v))
    stream = torch.cuda.Stream()
    stream.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(stream if warm else torch.cuda.current_stream()):
        want = [t.clone() for t in sb.attention_backward(q, k, v, o, lse, do, flags=4, **grads)]
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=stream):
        sb.attention_backward(q, k, v, o, lse, do, flags=4, **grads)
    with torch.cuda.stream(stream):
        sb.attention_backward(*big[:3], big_o, big_lse, big[3], flags=4)
        others = [torch.full((1 << n,), 3.0, device="cuda") for n in range(10, 21) for _ in range(4)]
    stream.synchronize()
    for t in grads.values():
        t.zero_()
    graph.replay()
    torch.cuda.synchronize()
    for got, ref in zip(grads.values(), want):
        assert torch.equal(got, ref)
    assert all(bool((t == 3).all()) for t in others) and sb.poll_device_status() == 0


@pytest.mark.parametrize("B,Hq,Hkv,S,D", [(24, 14, 2, 1024, 64), (3, 16, 4, 1237, 128)])
def test_reproducible_gradients_do_not_depend_on_the_chunks_of_the_host_call(sb, B, Hq, Hkv, S, D):
    """The first call is balanced with whole key tiles and its chunks are not; in the second the call and its chunks cut them."""
    from sentinel_b200 import _lib
    from sentinel_b200.host_pipeline import forward_backward_host
    g = torch.Generator().manual_seed(S)
    q, do, k, v = ((torch.randn(B, H, S, D, generator=g) * 0.5).to(torch.bfloat16).pin_memory() for H in (Hq, Hq, Hkv, Hkv))
    qd, dod, kd, vd = (t.cuda() for t in (q, do, k, v))
    o, lse = sb.attention_forward(qd, kd, vd)
    want = sb.attention_backward(qd, kd, vd, o, lse, dod, flags=_lib.FLAG_DETERMINISTIC)
    for got, ref in zip(forward_backward_host(q, k, v, do, flags=_lib.FLAG_DETERMINISTIC)[2:], want):
        assert torch.equal(got, ref.cpu())
    # with whole key tiles a sequence's gradients are the same bits whatever else is in the call
    flags = _lib.FLAG_DETERMINISTIC | _lib.FLAG_WHOLE_KEY_TILES
    want = sb.attention_backward(qd, kd, vd, o, lse, dod, flags=flags)
    alone = sb.attention_backward(*(t[1:2].contiguous() for t in (qd, kd, vd, o, lse, dod)), flags=flags)
    for got, ref in zip(alone, want):
        assert torch.equal(got, ref[1:2])
    assert sb.poll_device_status() == 0
