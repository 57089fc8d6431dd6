"""Which recurrences run as products over chunks: the rule alone, without a GPU."""
import math

import torch

BF16 = torch.bfloat16


class FakeLibrary:
    """Every entry is there; the ones that are called say how many bytes of scratch are needed."""

    def __init__(self, scratch=4096):
        self.scratch = scratch

    def __getattr__(self, name):
        def entry(*args):
            return self.scratch
        return entry


def fake_library(monkeypatch, ops, **kw):
    """The names of the kernels that are launched from here on."""
    seen, lib = [], FakeLibrary(**kw)
    monkeypatch.setattr(ops, "lib", lambda: lib)
    monkeypatch.setattr(ops, "_run", lambda name, fn, *args: seen.append(name))
    monkeypatch.setattr(ops, "_stream", lambda: None)
    monkeypatch.setattr(ops, "_ptr", lambda t: t)
    return seen


def test_scans_off_16_byte_boundaries_are_walked(monkeypatch):
    """Any buffer that the chunks read or write in whole pieces, four bytes off a boundary, keeps a
    step off them."""
    from binfer_b200.csrc import ops
    seen = fake_library(monkeypatch, ops)
    T, H, d = 400, 2, 8
    qs, slots = torch.tensor([0, T], dtype=torch.int32), torch.zeros(1, dtype=torch.int32)
    err = torch.zeros(1, dtype=torch.int32)

    def buf(*shape, off=False):
        n = math.prod(shape)
        x = torch.zeros(n + 8)
        at = (-x.data_ptr() // 4) % 4 + int(off)
        return x[at:at + n].view(*shape)

    def linear(off):
        ops.linear_scan(buf(T, 2, H, d, off=off == 0), buf(T, H, d, off=off == 1), buf(T, H),
                        buf(1, H * d * d), qs, slots, buf(T, H * d, off=off == 2), 1, H, H, d, d,
                        err, max_q=T, chunked=True)

    def retention(off):
        ops.retention_scan(torch.zeros(T, 3 * H * d), 0, H * d, 2 * H * d, buf(H), None, slots,
                           buf(1, H * d * d), qs, slots, buf(T, H * d, off=off == 2), 1, H, d, d, 1.0,
                           err, max_q=T, chunked=True)

    def mlstm(off):
        ops.mlstm_scan(torch.zeros(T, 4 * H * d, dtype=BF16), buf(T, 2 * H),
                       buf(1, H, ops.mlstm_state_size(d, d)), qs, slots,
                       buf(T, H * d, off=off == 2), 1, H, d, d, 1.0, err, max_q=T, chunked=True)

    def delta(off):
        ops.delta_scan(buf(T, 3 * H * d, off=off == 0), buf(T, 2, H), buf(1, H * d * d), qs, slots,
                       buf(T, H * d, off=off == 2), 1, H, H, d, d, err, max_q=T, chunked=True)

    for call, offs in ((linear, (0, 1, 2)), (retention, (2,)), (mlstm, (2,)), (delta, (0, 2))):
        seen.clear()
        call(None)
        assert any(n.endswith("_chunks") for n in seen), call
        for off in offs:
            seen.clear()
            call(off)
            assert seen and not any(n.endswith("_chunks") for n in seen), (call, off)
