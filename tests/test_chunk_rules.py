"""The recurrences as products over chunks, without a GPU: which ones run so, and the order of what no run shows."""
import math
import os
import re

import pytest
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
        ops.retention_scan(torch.zeros(T, 3 * H * d), 0, H * d, 2 * H * d, buf(H), None,
                           torch.arange(T, dtype=torch.int32),
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


def test_the_matrix_memory_asks_for_its_scratch_once(monkeypatch):
    """The room for a linear scan's terms is none of its business."""
    from binfer_b200.csrc import ops
    lib, asked = FakeLibrary(), []

    def entry(*args):
        asked.append(args[-1].value)
        return lib.scratch

    lib.bf_chunk_scan_scratch = entry
    monkeypatch.setattr(ops, "lib", lambda: lib)
    state = torch.zeros(1, 8, 256 * 512 + 512)
    for mlstm, want in ((1, [0]), (0, [1])):
        asked.clear()
        scratch, terms = ops._chunk_scratch(True, 2048, 2048, 1, 8, 8, 256, 512, state, mlstm)
        assert asked == want and terms == want[0] and scratch.numel() == 4096


# us on a B200: (heads, dk, dv, portions, tokens of each): (walk, products over chunks by multiply-adds, which the
# lines were laid by)
LINEAR_US = {
    (64, 128, 64, 1, 161): (42, 46), (64, 128, 64, 1, 200): (51, 50), (64, 128, 64, 1, 260): (64, 55),
    (64, 128, 64, 1, 1000): (232, 112), (64, 128, 64, 2, 161): (64, 65), (64, 128, 64, 2, 200): (76, 70),
    (64, 128, 64, 3, 161): (98, 74), (64, 128, 64, 12, 161): (310, 236), (8, 128, 256, 1, 161): (28, 39),
    (8, 128, 256, 1, 260): (41, 45), (8, 128, 256, 1, 350): (53, 46), (8, 128, 256, 2, 161): (41, 48),
    (8, 128, 256, 2, 220): (54, 49), (8, 128, 256, 3, 161): (52, 55), (8, 128, 256, 3, 220): (66, 60),
    (8, 128, 256, 6, 161): (98, 78), (8, 128, 256, 24, 161): (308, 238), (32, 64, 64, 1, 200): (28, 32),
    (32, 64, 64, 1, 500): (64, 38), (32, 64, 64, 2, 300): (40, 44), (32, 64, 64, 2, 500): (64, 50),
    (32, 64, 64, 6, 300): (75, 80), (32, 64, 64, 6, 400): (98, 101), (32, 64, 64, 6, 500): (122, 114),
    (32, 64, 64, 12, 260): (124, 133), (32, 64, 64, 12, 500): (237, 203), (32, 64, 64, 24, 240): (198, 203),
    (128, 128, 64, 1, 161): (65, 59), (128, 128, 64, 6, 161): (310, 230), (16, 128, 128, 1, 220): (35, 40),
    (16, 128, 128, 1, 350): (53, 47), (16, 128, 128, 2, 180): (46, 49), (16, 128, 128, 6, 180): (106, 78)}
DELTA_US = {
    (16, 128, 128, 1, 260): (74, 86), (16, 128, 128, 1, 400): (113, 97), (16, 128, 128, 2, 400): (144, 116),
    (16, 128, 128, 3, 400): (174, 200), (16, 128, 128, 3, 500): (217, 218), (16, 128, 128, 3, 700): (302, 275),
    (16, 128, 128, 6, 400): (342, 308), (16, 128, 128, 12, 400): (581, 566), (32, 128, 128, 1, 400): (144, 114),
    (32, 128, 128, 2, 400): (212, 216), (32, 128, 128, 2, 500): (265, 234), (32, 128, 128, 6, 500): (728, 646),
    (8, 128, 128, 3, 400): (144, 109), (8, 128, 128, 6, 400): (174, 200), (8, 128, 128, 6, 700): (302, 275),
    (16, 64, 64, 1, 400): (96, 77), (16, 64, 64, 2, 400): (96, 87), (16, 64, 64, 3, 400): (96, 110),
    (16, 64, 64, 3, 700): (165, 144), (16, 64, 64, 6, 700): (213, 279), (16, 64, 64, 6, 1000): (303, 385),
    (16, 64, 64, 12, 700): (270, 468), (16, 64, 64, 24, 350): (267, 509)}


@pytest.mark.parametrize("kind", ["linear", "delta"])
def test_the_rules_take_the_faster_way(kind):
    """At every measured point: within 8 % of the faster one, which is what runs of one side differ by
    and the points between which a line lies are apart."""
    from binfer_b200.csrc import ops
    rule, table = ((ops.chunk_scan_pays, LINEAR_US) if kind == "linear" else
                   (ops.delta_chunks_pay, DELTA_US))
    for (heads, dk, dv, portions, n), (walk, chunks) in table.items():
        pays = rule(portions * n, n, heads, dk, dv)
        assert (chunks if pays else walk) <= 1.08 * min(walk, chunks), (heads, dk, dv, portions, n)
        # single tokens beside the portions change little
        assert rule(portions * n + n // 50, n, heads, dk, dv) == pays


@pytest.mark.parametrize("positions", [None, torch.zeros(3, dtype=torch.int32)])
def test_retention_wants_a_position_per_row(monkeypatch, positions):
    from binfer_b200.csrc import ops
    seen = fake_library(monkeypatch, ops)
    one = torch.zeros(1, dtype=torch.int32)
    with pytest.raises(ops.KernelError, match="positions"):
        ops.retention_scan(torch.zeros(4, 24), 0, 8, 16, torch.zeros(1), None, positions,
                           torch.zeros(1, 64), one, one, torch.zeros(4, 8), 1, 1, 8, 8, 1.0, one)
    assert not seen


def test_a_chunks_flags_are_read_before_its_place_is_given_back():
    """ct_state's summing warps give a chunk's sums back by an arrival, and that is all that the flags of the chunk
    four further, in the same place, wait for: what is read behind it may be theirs.  (A run hardly ever shows it.)"""
    from binfer_b200.csrc import build
    with open(os.path.join(build.HERE, "chunk_tensor.cuh")) as f:
        kernel = f.read().split("ct_state_kernel(", 1)[1].split("\n}\n", 1)[0]
    sums = kernel[kernel.index("the state: key size"):]
    reads = [m.start() for m in re.finditer(r"odd_v\[", sums)]
    assert reads and sums.count("ct_arrive(sh.taken") == 1
    assert max(reads) < sums.index("ct_arrive(sh.taken")
