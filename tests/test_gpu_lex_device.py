"""ptxfe_lex_device_noalloc at the edges of its chunks, tiles and segments, at odd addresses, and with runs of soft bytes on
both sides of the tile kernels' look-back, against the ordinary lexer entry point."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

LINE = b"\tmad.lo.s32 %r12, %r3, 0x1F, -77; // c \"q\n"
SEGMENT = 4 << 20


def text_of(n, kind):
    if kind == "code":
        return (LINE * (n // len(LINE) + 1))[:n]
    body = (LINE * (n // len(LINE) + 1))[:n - 3000]
    return (body[:n // 2] + b" " + b"a1_" * 1000 + body[n // 2:])[:n]      # a run of soft bytes beyond the look-back


@pytest.mark.parametrize("n,kind", [(k, "code") for k in (1, 15, 31, 127, 128, 129, 8191, 8192, 8193, SEGMENT - 1, SEGMENT, SEGMENT + 1, 3 * SEGMENT + 4097)] +
                         [(20000, "run"), (SEGMENT + 9000, "run")])
@pytest.mark.parametrize("offset", [0, 1, 6])
def test_lex_device_edges(n, kind, offset):
    import torch
    import zluda_b200
    text = text_of(n, kind)
    ctx = zluda_b200.Context(0)
    want, errs = ctx.lex(text)
    ctx.close()
    lex = zluda_b200.lib().ptxfe_lex_device_noalloc
    lex.argtypes = [ctypes.c_int, ctypes.c_void_p, ctypes.c_uint64, ctypes.c_void_p, ctypes.c_uint64, ctypes.c_void_p, ctypes.c_void_p]
    buf = torch.full((n + offset,), ord("x"), dtype=torch.uint8, device="cuda")
    buf[offset:] = torch.frombuffer(bytearray(text), dtype=torch.uint8).cuda()
    for capacity in (len(want), len(want) // 2):
        tokens = torch.full((len(want) + 8,), -1, dtype=torch.int64, device="cuda")
        counts = torch.full((2,), -1, dtype=torch.int32, device="cuda")
        torch.cuda.synchronize()
        assert lex(0, buf.data_ptr() + offset, n, tokens.data_ptr(), capacity, counts.data_ptr(), None) == 0
        torch.cuda.synchronize()
        assert counts.tolist() == [len(want), len(errs)]
        got = tokens.cpu().numpy()
        assert (got[capacity:] == -1).all()
        w = got[:capacity].view(np.uint32).reshape(-1, 2)
        rows = np.array(want[:capacity], np.int64).reshape(-1, 3)
        assert (w[:, 0] == rows[:, 1]).all() and (w[:, 1] & 0xFFFF == rows[:, 2]).all() and (w[:, 1] >> 16 == rows[:, 0]).all()
