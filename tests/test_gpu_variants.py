"""Kernel variants chosen by a rule on sizes, at the edges of their ranges, against the oracle or the two-kernel path."""
import ctypes
import math

import pytest
import torch

from actlizela_b200.workloads import WORKLOADS, make_inputs
from oracle import gdn_oracle as oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m,k,n", [(1, 256, 8), (16, 264, 128), (17, 4096, 136), (32, 512, 2560), (33, 264, 264), (64, 4096, 128),
                                   (65, 1032, 2560), (128, 4096, 2560), (129, 4096, 1288), (300, 512, 2560), (896, 4096, 2560),
                                   (897, 4096, 2560)])
def test_out_proj_with_few_rows(m, k, n):
    """K split over a cluster: row counts at the edges of the 16/32/64/128-row tiles, ragged columns and K tails, and
    both sides of the rule that goes back to one CTA per tile."""
    from actlizela_b200 import out_proj_gemm
    gen = torch.Generator().manual_seed(m * 1000 + n)
    a = torch.randn(m, k, generator=gen).to(torch.bfloat16).cuda()
    w = (torch.randn(n, k, generator=gen) * k ** -0.5).to(torch.bfloat16).cuda()
    want = a.float() @ w.float().t()
    got = out_proj_gemm(a, w)
    assert got.shape == (m, n)
    assert oracle.rel_frobenius(got.float().cpu(), want.cpu()) < 3e-3
    assert oracle.max_abs(got.float(), want) <= 2 ** -8 * float(want.abs().max()) + 1e-6
    assert torch.equal(got, out_proj_gemm(a, w))                  # the sum over the cluster has one order


@pytest.mark.parametrize("m,k,n", [(13900, 72, 2504), (14001, 136, 2504), (2900, 72, 2504), (3001, 136, 2448), (5000, 64, 1288), (6000, 1024, 2560)])
def test_out_proj_square_tiles(m, k, n):
    """Tiles of 256 x 256 (the first two) and 256 x 224: rows that end in either 128-row half, columns that end in a
    box and in the 32 behind the boxes, one K step, a K tail, several turns.  An element is one
    BF16 rounding (2^-8 relative, two neighbours) from the FP32 sum; sums of K products differ by K 2^-24 of their terms."""
    from actlizela_b200 import out_proj_gemm
    gen = torch.Generator().manual_seed(m + k)
    a = torch.randn(m, k, generator=gen).to(torch.bfloat16).cuda()
    w = (torch.randn(n, k, generator=gen) * k ** -0.5).to(torch.bfloat16).cuda()
    want = a.double() @ w.double().t()
    got = out_proj_gemm(a, w)
    assert got.shape == (m, n)
    assert bool(((got.double() - want).abs() <= 2 ** -8 * want.abs() + 1e-4).all())


@pytest.mark.parametrize("m,k,n", [(1100, 264, 2560), (1930, 136, 2312), (2049, 72, 5128), (3000, 4096, 2560), (1999, 64, 5000)])
def test_out_proj_tile_widths(m, k, n):
    """Tiles of 128 and 256 columns, both sides of the rule: ragged rows, columns that end in either half of a wide tile,
    K of one step and with a tail."""
    from actlizela_b200 import out_proj_gemm
    gen = torch.Generator().manual_seed(m + n)
    a = torch.randn(m, k, generator=gen).to(torch.bfloat16).cuda()
    w = (torch.randn(n, k, generator=gen) * k ** -0.5).to(torch.bfloat16).cuda()
    want = a.float() @ w.float().t()
    got = out_proj_gemm(a, w)
    assert oracle.rel_frobenius(got.float().cpu(), want.cpu()) < 3e-3
    assert oracle.max_abs(got.float(), want) <= 2 ** -8 * float(want.abs().max()) + 1e-6


@pytest.mark.parametrize("batch,length,hk,hv", [(1, 1, 1, 1), (1, 64, 2, 6), (3, 129, 1, 2), (2, 193, 1, 4), (5, 700, 8, 32),
                                                (300, 65, 1, 1)])
def test_single_launch_form_equals_the_two_kernels_bitwise(batch, length, hk, hv, native_library):
    """One chunk, two, odd and even chunk counts, tails, several work items per CTA (more heads than SMs): the states
    and every output row have the bits of the two-kernel path."""
    from actlizela_b200.sm100 import Sm100Forward
    forward = Sm100Forward(native_library)
    w = WORKLOADS["cfg1"].sliced(batch=batch, length=length, key_heads=hk, value_heads=hv, seed=4000 + length)
    dev = [x.cuda() for x in make_inputs(w)]
    want_out, want_state = forward(*dev, True, configuration="umma")
    out, state = forward(*dev, True, configuration="fused")
    torch.cuda.synchronize()
    assert _healthy(native_library)
    assert torch.equal(out, want_out) and torch.equal(state, want_state)
    out_only, none = forward(*dev, False, configuration="fused")
    assert none is None and torch.equal(out_only, want_out)


@pytest.mark.parametrize("length,hv", [(64 * 110 + 1, 4), (64 * 89, 5)])
@pytest.mark.parametrize("raw", [False, True])
def test_both_occupancies_of_the_prepare_kernel(length, hv, raw, native_library):
    """444 blocks, one turn of three CTAs an SM, and 445, which four take: the single launch's bits, from prepared tensors and
    from raw projections (two kernels against the same in three launches)."""
    from actlizela_b200 import gdn_forward_projections, gdn_prepare_inputs
    from actlizela_b200.sm100 import Sm100Forward
    forward = Sm100Forward(native_library)
    if raw:
        gen = torch.Generator().manual_seed(length)
        mixed = torch.randn(1, length, (2 + hv) * 128, generator=gen).to(torch.bfloat16).cuda()
        a, b = (torch.randn(1, length, hv, generator=gen).to(torch.bfloat16).cuda() for _ in range(2))
        a_log, dt_bias = torch.zeros(hv, device="cuda"), torch.full((hv,), -8.0, device="cuda")       # slow: two kernels
        q, k, v, g, beta = (x.unsqueeze(0) for x in gdn_prepare_inputs(mixed[0], a[0], b[0], a_log, dt_bias, 1, hv))
        out, state = gdn_forward_projections(mixed, a, b, a_log, dt_bias, 1, hv, None)
    else:
        w = WORKLOADS["cfg1"].sliced(batch=1, length=length, key_heads=1, value_heads=hv, seed=length)
        q, k, v, g, beta, _ = [x.cuda() if x is not None else None for x in make_inputs(w)]
        out, state = forward(q, k, v, g, beta, None, True, configuration="umma")
    want_out, want_state = forward(q, k, v, g, beta, None, True, configuration="fused")
    torch.cuda.synchronize()
    assert _healthy(native_library)
    assert torch.equal(out, want_out) and torch.equal(state, want_state)


def _healthy(native_library):
    status = (ctypes.c_int * 4)()
    return native_library.lib.actlize_la_sm100_device_status(status, 1) == 0 and status[0] == 0


@pytest.mark.parametrize("batch,length,hk,hv", [(1, 64 * 16, 1, 2), (1, 64 * 17 + 5, 2, 6), (2, 64 * 40 + 1, 1, 2), (1, 64 * 300 + 1, 1, 1),
                                                (1, 64 * 1300, 1, 2), (1, 64 * 20 + 63, 37, 74)])
@pytest.mark.parametrize("stress", ["none", "slow-head", "long-key"])
def test_heads_cut_over_the_sms(batch, length, hk, hv, stress, native_library):
    """Heads cut into two pieces up to one for every SM, of the least length and of many chunks: agreement with the
    unsplit walk to exp(-40) of the state, and a head whose gates hardly decay or that holds a token that is no
    contraction comes out with the unsplit walk's bits."""
    from actlizela_b200.sm100 import Sm100Forward
    forward = Sm100Forward(native_library)
    w = WORKLOADS["cfg1"].sliced(batch=batch, length=length, key_heads=hk, value_heads=hv, seed=5000 + length)
    q, k, v, g, beta, init = make_inputs(w)
    lone = hv - 1
    if stress == "slow-head":
        g[:, :, lone] *= 1e-3
    elif stress == "long-key":
        beta[:, length - 3, lone] = -0.25
    dev = [x.cuda() for x in (q, k, v, g, beta, init)]
    want_out, want_state = forward(*dev, True, configuration="fused")
    counts = (ctypes.c_int * 2)()
    assert native_library.lib.actlize_la_sm100_walk_plan_counts(counts, 1) == 0
    out, state = forward(*dev, True, configuration="fused-split")
    torch.cuda.synchronize()
    assert _healthy(native_library)
    assert native_library.lib.actlize_la_sm100_walk_plan_counts(counts, 1) == 0
    alone = 0 if stress == "none" else batch
    assert list(counts) == [batch * hv - alone, alone]
    assert oracle.max_abs(out.float(), want_out.float()) < 1e-5
    assert oracle.rel_frobenius(state.cpu(), want_state.cpu()) < 1e-6
    if stress != "none":
        assert torch.equal(out[:, :, lone], want_out[:, :, lone]) and torch.equal(state[:, lone], want_state[:, lone])
    again_out, again_state = forward(*dev, True, configuration="fused-split")
    assert torch.equal(again_out, out) and torch.equal(again_state, state)


@pytest.mark.parametrize("sequences,hv", [(149, 1), (75, 2), (256, 1), (257, 1)])
def test_packed_sequences_dealt_longest_first(sequences, hv, native_library):
    """More packed sequences than SMs, up to the most that are ordered and one more, some empty: the bits of calls that hold
    too few sequences to be ordered."""
    from actlizela_b200 import gdn_forward_varlen
    lengths = [(37 * i * i + 11 * i) % 190 for i in range(sequences)]
    bounds = [0]
    for n in lengths:
        bounds.append(bounds[-1] + n)
    w = WORKLOADS["cfg1"].sliced(batch=1, length=bounds[-1], key_heads=1, value_heads=hv, seed=6000 + sequences)
    q, k, v, g, beta, _ = (x.cuda() if x is not None else None for x in make_inputs(w))
    init = torch.randn(sequences, hv, 128, 128, device="cuda") * 0.05
    out, state = gdn_forward_varlen(q, k, v, g, beta, torch.tensor(bounds, dtype=torch.int32, device="cuda"), init, True)
    for first in range(0, sequences, 70):
        last = min(first + 70, sequences)
        a, b = bounds[first], bounds[last]
        part = [x[:, a:b].contiguous() for x in (q, k, v, g, beta)]
        offsets = torch.tensor([x - a for x in bounds[first:last + 1]], dtype=torch.int32, device="cuda")
        want_out, want_state = gdn_forward_varlen(*part, offsets, init[first:last].contiguous(), True)
        assert torch.equal(out[:, a:b], want_out) and torch.equal(state[first:last], want_state)


@pytest.mark.parametrize("lengths,hv", [([1], 1), ([0, 0, 577, 0, 63, 64, 65, 0], 6), ([300, 1, 129, 700] * 11, 1), ([640] * 44, 2),
                                        ([255] * 25, 2), ([230] * 25, 2), ([2000, 3], 44)])
def test_packed_sequences_in_two_kernels(lengths, hv, native_library):
    """Few packed sequences, both sides of the rule, empty and ragged ones: the bits of the fixed-shape forward.  Device offsets
    that run back or past the tensors mean what their clamped values mean."""
    from actlizela_b200 import gdn_forward_varlen
    bounds = [0]
    for n in lengths:
        bounds.append(bounds[-1] + n)
    w = WORKLOADS["cfg1"].sliced(batch=1, length=bounds[-1], key_heads=1, value_heads=hv, seed=8000 + bounds[-1])
    q, k, v, g, beta, _ = (x.cuda() if x is not None else None for x in make_inputs(w))
    init = 0.05 * torch.randn(len(lengths), hv, 128, 128, generator=torch.Generator().manual_seed(len(lengths))).cuda()
    want_out, want_state = gdn_forward_varlen(q, k, v, g, beta, bounds, init, True, per_sequence=True, algorithm="wy_sm100",
                                              backend="cuda_sm100", configuration="umma")
    for initial in (init, None):
        out, state = gdn_forward_varlen(q, k, v, g, beta, torch.tensor(bounds, dtype=torch.int32, device="cuda"), initial, True)
        torch.cuda.synchronize()
        assert _healthy(native_library)
        if initial is not None:
            assert torch.equal(out, want_out) and torch.equal(state, want_state)
    host_out, host_state = gdn_forward_varlen(q, k, v, g, beta, bounds, init, True)
    assert torch.equal(host_out, want_out) and torch.equal(host_state, want_state)
    odd = [1 << 30 if i == len(lengths) else at - 5 * (i % 3) for i, at in enumerate(bounds)]
    clean, most = [0], 0
    for at in odd[1:]:
        most = max(most, at)
        clean.append(min(most, bounds[-1]))
    odd_out, odd_state = gdn_forward_varlen(q, k, v, g, beta, torch.tensor(odd, dtype=torch.int32, device="cuda"), init, True)
    want_out, want_state = gdn_forward_varlen(q, k, v, g, beta, clean, init, True)
    assert torch.equal(odd_out, want_out) and torch.equal(odd_state, want_state)


@pytest.mark.parametrize("chunks,reach,split", [
    (300, (4, 20, 60), 2),                   # too slow for 37 pieces in the single launch, two of them not for eight
    (300, (30, 20, 12, 36, 1000), 4),
    (131, (9, 17, 25), 1),                   # pieces of 8, and of 16 chunks: the first just too slow for the former
    (130, (2, 3, 64, 65), 2)])
def test_cuts_follow_the_gates(chunks, reach, split, native_library):
    """Heads whose state outlives the shortest pieces, each by another factor: where the single launch's pieces are too short for
    one, all are cut into eight in the two kernels, or walked whole with the unsplit walk's bits.  Under slow gates a piece's own rounding (16-bit operand pairs: the
    state is good to 4e-6) is not forgotten within the piece: both walks' errors in the state, and single BF16 flips in the
    output, which has 2^-9 per flipped value (a sixteenth of them is 5e-4)."""
    from actlizela_b200.sm100 import Sm100Forward
    forward = Sm100Forward(native_library)
    length, hv = 64 * chunks - 7, len(reach)
    w = WORKLOADS["cfg1"].sliced(batch=1, length=length, key_heads=1, value_heads=hv, seed=7000 + chunks)
    q, k, v, g, beta, init = make_inputs(w)
    gen = torch.Generator().manual_seed(chunks)
    for h, r in enumerate(reach):            # 40 nats within r chunks, with half a chunk to spare
        g[:, :, h] = -40.0 / (64 * (r - 0.5)) * (0.9 + 0.2 * torch.rand(1, length, generator=gen))
    dev = [x.cuda() for x in (q, k, v, g, beta, init)]
    want_out, want_state = forward(*dev, True, configuration="fused")
    counts = (ctypes.c_int * 2)()
    assert native_library.lib.actlize_la_sm100_walk_plan_counts(counts, 1) == 0
    out, state = forward(*dev, True, configuration="fused-split")
    torch.cuda.synchronize()
    assert _healthy(native_library)
    assert native_library.lib.actlize_la_sm100_walk_plan_counts(counts, 1) == 0
    assert list(counts) == [split, hv - split]
    for h in range(hv):
        assert oracle.rel_frobenius(out[:, :, h].float().cpu(), want_out[:, :, h].float().cpu()) < 5e-4
        assert oracle.rel_frobenius(state[:, h].cpu(), want_state[:, h].cpu()) < 8e-6
    for h, r in enumerate(reach):
        if r > chunks:
            assert torch.equal(out[:, :, h], want_out[:, :, h]) and torch.equal(state[:, h], want_state[:, h])
    again_out, again_state = forward(*dev, True, configuration="fused-split")
    assert torch.equal(again_out, out) and torch.equal(again_state, state)


@pytest.mark.parametrize("batch,length,hk,hv,slow,split", [
    (1, 64, 1, 2, {}, None),                             # one chunk: single launch
    (1, 65, 1, 2, {}, None),
    (1, 700, 2, 8, {}, None),                            # few heads: two kernels, walked whole
    (3, 64 * 9 + 1, 1, 2, {}, None),                     # rows behind a batch element's end are the next one's
    (1, 64 * 60 + 9, 2, 8, {}, 8),                       # cut into seven
    (1, 64 * 60 + 9, 2, 8, {3: 7, 5: 1000}, 7),          # one head that just allows that, one that does not
    (1, 64 * 180 + 9, 2, 8, {}, 8),                      # single launch, cut into 18
    (1, 64 * 180 + 9, 2, 8, {3: 18, 5: 1000}, 7),        # left to the two kernels: cut into eight, one head walked whole
    (2, 64 * 250, 3, 6, {4: 60}, 10),
    (2, 64 * 16 + 3, 37, 37, {3: 1000}, 72),             # the most heads that can be cut, into two
    (5, 64 * 2 + 3, 5, 15, {}, None)])                   # one head more: single launch
def test_projections_in_every_form(batch, length, hk, hv, slow, split, native_library):
    """Raw projections in the two kernels (one CTA per key head stores its normalised queries and keys), walked whole and cut, in
    the single launch, and left by it: the outputs of prepare_inputs + forward, bit for bit where that walks them alike.  ``slow``:
    chunks that a head's state outlives."""
    from actlizela_b200 import gdn_forward_projections, gdn_prepare_inputs
    from actlizela_b200.sm100 import Sm100Forward
    gen = torch.Generator().manual_seed(9000 + length)
    mixed = torch.randn(batch, length, (2 * hk + hv) * 128, generator=gen).to(torch.bfloat16).cuda()
    a, b = ((0.1 * torch.randn(batch, length, hv, generator=gen)).to(torch.bfloat16).cuda() for _ in range(2))
    a_log, dt_bias = torch.zeros(hv), torch.zeros(hv)
    for h, reach in slow.items():                        # softplus(0) = 0.693 nats a token, scaled
        a_log[h] = math.log(40.0 / (64 * (reach - 0.5)) / 0.693)
    a_log, dt_bias = a_log.cuda(), dt_bias.cuda()
    initial = (0.05 * torch.randn(batch, hv, 128, 128, generator=gen)).cuda()
    rows = batch * length
    prepared = [x.view(batch, length, *x.shape[1:]) for x in
                gdn_prepare_inputs(mixed.view(rows, -1), a.view(rows, hv), b.view(rows, hv), a_log, dt_bias, hk, hv)]
    want_out, want_state = Sm100Forward(native_library)(*prepared, initial, True, configuration="umma")
    counts = (ctypes.c_int * 2)()
    assert native_library.lib.actlize_la_sm100_walk_plan_counts(counts, 1) == 0
    out, state = gdn_forward_projections(mixed, a, b, a_log, dt_bias, hk, hv, initial, True)
    torch.cuda.synchronize()
    assert _healthy(native_library)
    assert native_library.lib.actlize_la_sm100_walk_plan_counts(counts, 1) == 0
    if split is not None:
        assert list(counts) == [split, batch * hv - split]
    for h in range(hv):
        if split is None or slow.get(h) == 1000:
            assert torch.equal(out[:, :, h], want_out[:, :, h]) and torch.equal(state[:, h], want_state[:, h])
        else:                                            # as in test_cuts_follow_the_gates
            assert oracle.rel_frobenius(out[:, :, h].float().cpu(), want_out[:, :, h].float().cpu()) < 5e-4
            assert oracle.rel_frobenius(state[:, h].cpu(), want_state[:, h].cpu()) < 8e-6


def test_static_scratch_takes_cut_heads_at_its_limit(native_library):
    """64 blocks, the most the built-in array is for, in the form that needs words in front of the factors."""
    from tests.test_zz_no_alloc import _call
    w = WORKLOADS["cfg1"].sliced(batch=1, length=64 * 64, key_heads=1, value_heads=1, seed=64)
    dev = [x.cuda() for x in make_inputs(w)]
    from actlizela_b200.sm100 import Sm100Forward
    want_out, want_state = Sm100Forward(native_library)(*dev, True, configuration="fused-split")
    rc, out, state = _call(native_library.lib, dev, config=4 | (8 << 16))
    torch.cuda.synchronize()
    assert rc == 0 and _healthy(native_library)
    assert torch.equal(out, want_out) and torch.equal(state, want_state)


@pytest.mark.parametrize("call", ["cut", "left", "raw-two-kernels", "raw-cut", "raw-left", "packed-two-kernels"])
def test_forms_under_capture_and_on_a_side_stream(call, native_library):
    """Every chain of launches captured into a graph and replayed on other inputs in the same buffers, the flags and the scan's
    words of the capture among them: the eager call's bits."""
    from actlizela_b200 import gdn_forward, gdn_forward_projections, gdn_forward_varlen
    gen = torch.Generator(device="cuda").manual_seed(17)
    draw = lambda *shape: torch.randn(*shape, generator=gen, device="cuda")
    norm = lambda x: torch.nn.functional.normalize(x, dim=-1).to(torch.bfloat16)

    def inputs(slow):
        if call.startswith("raw"):
            t, hk, hv = (700, 2, 4) if call == "raw-two-kernels" else (64 * 250, 2, 6)
            bias = torch.zeros(hv, device="cuda")
            if slow:
                bias[1] = -12.0
            return [draw(1, t, (2 * hk + hv) * 128).to(torch.bfloat16), draw(1, t, hv).to(torch.bfloat16), draw(1, t, hv).to(torch.bfloat16),
                    torch.zeros(hv, device="cuda"), bias]
        t, hk, hv = (1500, 1, 2) if call.startswith("packed") else (64 * 180, 2, 8)
        g = -torch.rand(1, t, hv, generator=gen, device="cuda")
        if slow:
            g[:, :, 1] *= 1e-4
        return [norm(draw(1, t, hk, 128)), norm(draw(1, t, hk, 128)), draw(1, t, hv, 128).to(torch.bfloat16), g,
                torch.sigmoid(draw(1, t, hv)).to(torch.bfloat16)]

    slow = call.endswith("left")
    x, other = inputs(slow), inputs(slow)
    if call.startswith("packed"):
        x.append(torch.tensor([0, 100, 100, 900, 1500], dtype=torch.int32, device="cuda"))
        other.append(torch.tensor([0, 64, 640, 641, 1500], dtype=torch.int32, device="cuda"))
        run = lambda a: gdn_forward_varlen(*a[:5], a[5], None, True)
    elif call.startswith("raw"):
        run = lambda a: gdn_forward_projections(*a, 2, a[3].numel(), None, True)
    else:
        run = lambda a: gdn_forward(*a, None, True)
    want, want_other = run(x), run(other)
    stream = torch.cuda.Stream()
    stream.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(stream):
        beside = run(x)
    torch.cuda.current_stream().wait_stream(stream)
    assert torch.equal(beside[0], want[0]) and torch.equal(beside[1], want[1])
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        got = run(x)
    for values, wanted in ((x, want), (other, want_other), ([y.clone() for y in inputs(not slow)] + x[5:], None)):
        wanted = wanted or run(values)
        for slot, value in zip(x, [y.clone() for y in values]):
            slot.copy_(value)
        graph.replay()
        torch.cuda.synchronize()
        assert _healthy(native_library)
        assert torch.equal(got[0], wanted[0]) and torch.equal(got[1], wanted[1])
