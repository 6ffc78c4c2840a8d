"""Work buffers between contexts: handed from a context on one stream to one on another, and left alone by captures."""
import threading

import pytest
import torch

pytestmark = pytest.mark.gpu
SCALE = 192.0 ** -0.5


def _problem(seed, B, T):
    g = torch.Generator(device="cuda").manual_seed(seed)

    def rn(*s):
        return torch.randn(*s, device="cuda", generator=g).to(torch.bfloat16)
    return rn(B, 64, 576), rn(B, T, 576), torch.full((B,), T, dtype=torch.int32, device="cuda"), T


def _decode(attn, p, out=None):
    return attn.mla_decode(p[0], p[1], p[2], max_kv_len=p[3], scale=SCALE, out=out)


def test_a_buffer_goes_from_one_stream_to_another():
    """A context is closed with its calls still running, and the next one, on another stream, starts at once: each gets its
    own split records, whoever had the buffer before. The same bytes as alone."""
    from cwick_b200.ops import Attn
    first, second = _problem(1, 8, 16384), _problem(2, 4, 8192)
    alone = Attn(0)
    want = [_decode(alone, p) for p in (first, second)]
    torch.cuda.synchronize()
    streams = [torch.cuda.Stream() for _ in range(2)]
    for _ in range(4):
        got = []
        for s, p in zip(streams, (first, second)):
            with torch.cuda.stream(s):
                a = Attn(0)
                outs = [_decode(a, p) for _ in range(8)]
                a.ctx.close()
                got.append(outs)
        torch.cuda.synchronize()
        for outs, w in zip(got, want):
            assert all(torch.equal(o, w) for o in outs)


@pytest.mark.parametrize("what", ["close", "grow"])
def test_another_threads_capture_survives(what):
    """One thread captures a call; meanwhile another closes a context, or calls one with a longer input so that its buffers
    grow. The capture ends well and its graph gives the call's result."""
    from cwick_b200.ops import Attn
    small, large = _problem(3, 1, 4096), _problem(4, 8, 32768)
    s, side = torch.cuda.Stream(), torch.cuda.Stream()
    with torch.cuda.stream(side):
        other = Attn(0)
        want_large = _decode(Attn(0), large)
        _decode(other, small)
        out_large = torch.empty_like(want_large)
    with torch.cuda.stream(s):
        attn = Attn(0)
        want = _decode(attn, small).clone()
        out = torch.empty_like(want)
        torch.cuda.synchronize()
        failed = []

        def meanwhile():
            try:
                if what == "close":
                    other.ctx.close()
                else:
                    with torch.cuda.stream(side):
                        _decode(other, large, out_large)
            except Exception as e:                       # noqa: BLE001 -- shown by the main thread
                failed.append(e)
        graph = torch.cuda.CUDAGraph()
        graph.capture_begin(capture_error_mode="thread_local")
        try:
            _decode(attn, small, out)
            t = threading.Thread(target=meanwhile)
            t.start()
            t.join()
        finally:
            graph.capture_end()
        assert not failed, failed
        graph.replay()
        torch.cuda.synchronize()
        assert torch.equal(out, want)
        if what == "grow":
            assert torch.equal(out_large, want_large)
        del graph
