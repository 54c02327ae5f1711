"""The device-buffer operator called on several streams of one context: every call
computes its own block, whatever the calls around it stage."""
import ctypes

import pytest

import oracle
from oracle import Geom

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def gb():
    import granite_b200
    return granite_b200


def _block(gb, o, n, seed):
    import torch
    g = Geom(n, tuple(-0.125 * a for a in n), tuple(0.125 * a for a in n))
    u = oracle.add_noise(o.init_brill_lindquist(g, [1.0], [[0.12, -0.1, 0.05]], r_floor=0.5 * g.dx[0]), 1e-10, seed)
    return gb.GridBlock(0, 0, g.n, g.lo, g.hi).desc(), torch.from_numpy(u).cuda()


def _call(op, desc, u, rhs, stream):
    op.ctx.check(op.ctx.lib.granite_ccz4_compute_rhs_device(
        op.ctx.h, ctypes.byref(desc), ctypes.c_void_p(u.data_ptr()), ctypes.c_void_p(rhs.data_ptr()), None, None, None,
        None, op.precision, ctypes.c_void_p(stream) if stream else None))


# a long launch and short ones, with and without tensor maps (odd row length); the
# context's own stream (None) among the callers'
@pytest.mark.parametrize("precision", [0, 1])
def test_calls_on_two_streams_keep_their_blocks(gb, oracle_lib, precision):
    import torch
    op = gb.CCZ4Evolution(gb.CCZ4Params(), precision)
    blocks = [_block(gb, oracle_lib, n, 3 + i) for i, n in enumerate([(96, 64, 48), (24, 20, 16), (27, 13, 9)])]
    want = []
    for desc, u in blocks:
        rhs = torch.zeros_like(u)
        torch.cuda.synchronize()
        _call(op, desc, u, rhs, None)
        op.ctx.check(op.ctx.lib.granite_ccz4_sync(op.ctx.h))
        want.append(rhs)
    streams = [torch.cuda.Stream().cuda_stream, torch.cuda.Stream().cuda_stream, None]
    outs = [[torch.zeros_like(u) for _, u in blocks] for _ in range(12)]
    torch.cuda.synchronize()
    for k, out in enumerate(outs):
        for i, (desc, u) in enumerate(blocks):
            _call(op, desc, u, out[i], streams[(k + 2 * i + k // 3) % 3])
    op.ctx.check(op.ctx.lib.granite_ccz4_sync(op.ctx.h))
    torch.cuda.synchronize()
    for out in outs:
        for i in range(len(blocks)):
            assert torch.equal(out[i], want[i]), f"block {i}"


def test_a_stream_of_the_same_handle_is_another_stream(gb, oracle_lib):
    # streams made and destroyed around every call: a handle may come again
    import torch
    rt = torch.cuda.cudart()
    op = gb.CCZ4Evolution(gb.CCZ4Params())
    blocks = [_block(gb, oracle_lib, n, 5 + i) for i, n in enumerate([(64, 64, 48), (24, 20, 16)])]
    outs = [torch.zeros_like(blocks[k % 2][1]) for k in range(10)]
    torch.cuda.synchronize()
    for k, out in enumerate(outs):
        handle = ctypes.c_void_p()
        assert int(rt.cudaStreamCreate(ctypes.addressof(handle))) == 0
        _call(op, *blocks[k % 2], out, handle.value)
        assert int(rt.cudaStreamDestroy(handle.value)) == 0  # (its work still runs to the end)
    torch.cuda.synchronize()
    for k in range(2, 10):
        assert torch.equal(outs[k], outs[k % 2])
    assert torch.count_nonzero(outs[0]) and torch.count_nonzero(outs[1])
