"""One pass over the weights for 3 to 16 batch rows (gemv_rows_kernel) against the oracle."""
import numpy as np
import pytest
import torch

import oracle
from eptq_b200 import _lib
from eptq_b200.kernels.linear import EPTQLinear, forward_group
from eptq_b200.synthetic import make_activations, make_layer
from tests import util

pytestmark = pytest.mark.gpu
DEV = "cuda"
TABLES = {"e8_d4": oracle.d4_table(1.75), "e8_lattice": oracle.e8_table(1.6)}


def layers_of(kind, shapes, fractions=(0.004, 0.0, 0.02)):
    qds = [make_layer(o, i, seed=7 * k + o + i, outlier_frac=fractions[k % len(fractions)], bias=(k % 2 == 0))
           for k, (o, i) in enumerate(shapes)]
    return qds, [EPTQLinear.from_quantized_data(qd, torch.from_numpy(TABLES[kind]), kind).to(DEV) for qd in qds]


def check(kind, qds, xs, ys):
    for qd, x, y in zip(qds, xs, ys):
        W16 = oracle.dequantize_layer(util.qld_arrays(qd), TABLES[kind])
        ref = oracle.linear_reference(x.numpy(), W16, None if qd.bias is None else qd.bias.numpy())
        for b in range(x.shape[0]):                     # row by row: rows may differ in scale
            assert util.max_rel_err(y[b].float().cpu().numpy(), ref[b]) <= util.REL_TOL


@pytest.mark.parametrize("kind", ["e8_d4", "e8_lattice"])
@pytest.mark.parametrize("batch", [3, 4, 5, 8, 9, 16])
def test_rows_match_oracle(kind, batch):
    # shares that begin and end inside row tiles, ragged row counts, one row, one 32-column step, layers without
    # critical blocks between layers with them
    shapes = [(1288, 2752), (264, 4096), (8, 32), (4096, 1056), (40, 96)]
    qds, lins = layers_of(kind, shapes)
    xs = [make_activations(batch, i, seed=61 + k) * (10.0 ** (k % 3 - 1)) for k, (_, i) in enumerate(shapes)]
    for _ in range(2):                                  # the scratch is left clean
        ys = forward_group(lins, [x.to(DEV) for x in xs])
        check(kind, qds, xs, ys)
    first = forward_group(lins, [x.to(DEV) for x in xs])
    again = forward_group(lins, [x.to(DEV) for x in xs])
    assert all(torch.equal(a, b) for a, b in zip(first, again))          # partials are added in a fixed order


@pytest.mark.parametrize("kind", ["e8_d4", "e8_lattice"])
def test_rows_many_layers_and_all_markers(kind):
    qds, lins = layers_of(kind, [(64, 64 + 32 * (k % 5)) for k in range(32)])
    qds[3] = make_layer(64, qds[3].Q.shape[1], seed=5, outlier_frac=1.1)                 # nothing but critical blocks
    lins[3] = EPTQLinear.from_quantized_data(qds[3], torch.from_numpy(TABLES[kind]), kind).to(DEV)
    lins[3]._codebook = lins[0]._codebook
    lins[3]._codebook32 = lins[0]._codebook32
    xs = [make_activations(6, qd.Q.shape[1], seed=9 + k) for k, qd in enumerate(qds)]
    check(kind, qds, xs, forward_group(lins, [x.to(DEV) for x in xs]))


@pytest.mark.parametrize("kind", ["e8_d4", "e8_lattice"])
def test_small_scratch_takes_passes_of_two_rows(kind):
    """A caller whose scratch holds no partial sums still gets its result."""
    import ctypes as C
    qds, lins = layers_of(kind, [(4096, 1024), (1024, 1024)])
    x = make_activations(7, 1024, seed=3)
    xd = x.to(DEV)
    lib = _lib.load()
    descs = (_lib.EptqLayer * 2)(*[lin.descriptor() for lin in lins])
    assert lib.eptq_group_workspace_bytes(C.byref(descs), 2, 7) > 1 << 20
    ws = torch.zeros(1 << 20, dtype=torch.uint8, device=DEV)
    ys = [torch.empty((7, lin.out_features), dtype=torch.float16, device=DEV) for lin in lins]
    xp = (C.c_void_p * 2)(xd.data_ptr(), xd.data_ptr())
    yp = (C.c_void_p * 2)(*[y.data_ptr() for y in ys])
    st = lib.eptq_linear_forward_group(C.byref(descs), 2, xp, yp, 7, ws.data_ptr(), ws.numel(),
                                       torch.cuda.current_stream().cuda_stream)
    assert st == 0
    check(kind, qds, [x, x], ys)


@pytest.mark.parametrize("kind", ["e8_d4", "e8_lattice"])
@pytest.mark.parametrize("out,inn,qb,batch", [(4096, 6176, 128, 1), (5120, 5504, 512, 3), (4160, 4128, 64, 5), (4096, 6176, 2048, 16)])
def test_group_scales_match_oracle(kind, out, inn, qb, batch):
    """Group scales in passes of four rows; scales that span a factor of about a thousand."""
    from eptq_b200.kernels import h_absmax
    qd = make_layer(out, inn, seed=out + qb, outlier_frac=0.01, bias=(batch % 2 == 1), qb_size=qb)
    gen = torch.Generator().manual_seed(qb)
    qd.S_group = torch.exp(1.2 * torch.randn(qd.S_group.shape, generator=gen)).to(torch.float16)
    lin = EPTQLinear.from_quantized_data(qd, torch.from_numpy(TABLES[kind]), kind).to(DEV)
    x = make_activations(batch, inn, seed=qb + batch)
    before = _lib.load().eptq_kernel_launch_count(1)
    y = lin(x.to(DEV))
    torch.cuda.synchronize()
    assert _lib.load().eptq_kernel_launch_count(1) - before == (batch + 3) // 4       # the multi-row kernel took it
    assert lin.descriptor().h_absmax == pytest.approx(-h_absmax(lin.h) * h_absmax(lin.S_group))
    W16 = oracle.dequantize_layer(util.qld_arrays(qd), TABLES[kind])
    ref = oracle.linear_reference(x.numpy(), W16, None if qd.bias is None else qd.bias.numpy())
    for b in range(batch):
        assert util.max_rel_err(y[b].float().cpu().numpy(), ref[b]) <= util.REL_TOL


@pytest.mark.parametrize("kind", ["e8_d4", "e8_lattice"])
def test_group_scales_written_just_before_the_call(kind):
    """A layer with group scales sees what the kernel before it on the stream wrote to any of its weights."""
    import ctypes as C
    lib = _lib.load()
    lins, want = [], []
    x = make_activations(1, 6176, seed=3).to(DEV)
    for seed in (1, 2):
        qd = make_layer(4096, 6176, seed=seed, outlier_frac=0.0, qb_size=128)
        lins.append(EPTQLinear.from_quantized_data(qd, torch.from_numpy(TABLES[kind]), kind).to(DEV))
        want.append(lins[-1](x))
    target = EPTQLinear.from_quantized_data(make_layer(4096, 6176, seed=1, outlier_frac=0.0, qb_size=128),
                                            torch.from_numpy(TABLES[kind]), kind).to(DEV)
    d = target.descriptor()
    d.h_absmax = min(lin.descriptor().h_absmax for lin in lins)               # bounds either layer's scales
    ws = torch.zeros(lib.eptq_layer_workspace_bytes(C.byref(d), 1), dtype=torch.uint8, device=DEV)
    ys = [torch.empty_like(want[0]) for _ in range(16)]
    for n, y in enumerate(ys):
        for name in ("S_group", "h", "g", "Q"):
            getattr(target, name).copy_(getattr(lins[n % 2], name))
        assert lib.eptq_linear_forward(C.byref(d), x.data_ptr(), y.data_ptr(), 1, ws.data_ptr(), ws.numel(),
                                       torch.cuda.current_stream().cuda_stream) == 0
    for n, y in enumerate(ys):
        ref = want[n % 2].float()
        assert torch.allclose(y.float(), ref, rtol=2e-3, atol=2e-3 * float(ref.abs().max()))


@pytest.mark.parametrize("kind,out,inn,frac", [("e8_d4", 1024, 4096, 0.002), ("e8_d4", 512, 4096, 0.02), ("e8_lattice", 1024, 8192, 0.002)])
@pytest.mark.parametrize("batch", [3, 8, 16])
def test_rows_few_tiles(kind, out, inn, frac, batch):
    """Many blocks with short shares per row tile: a unit of corrections often takes the tile's last ticket."""
    qds, lins = layers_of(kind, [(out, inn)], (frac,))
    x = make_activations(batch, inn, seed=batch)
    ys = [lins[0](x.to(DEV)) for _ in range(20)]
    check(kind, qds, [x], ys[:1])
    assert all(torch.equal(y, ys[0]) for y in ys)


@pytest.mark.parametrize("kind", ["e8_d4", "e8_lattice"])
@pytest.mark.parametrize("spread_s,spread_h", [(0.1, 0.25), (1.2, 0.1)])
def test_group_scales_keep_32_bits(kind, spread_s, spread_h):
    """Activations of any size, each batch row its own, and scales that differ a thousandfold between groups.  The sums are
    compared beyond fp16 by a second call whose bias cancels the first one's result."""
    out, inn, qb = 4096, 6176, 128
    gen = torch.Generator(device=DEV).manual_seed(11)
    qd = make_layer(out, inn, seed=4, outlier_frac=0.004, qb_size=qb, device=DEV, scale_sigma=spread_h)
    qd.S_group = torch.exp(spread_s * torch.randn(qd.S_group.shape, generator=gen, device=DEV)).half()
    lin = EPTQLinear.from_quantized_data(qd, torch.from_numpy(TABLES[kind]).to(DEV), kind)
    code = lin._codebook32.double()
    idx = lin.Q.long() + 32768
    if kind == "e8_d4":
        W = torch.cat([code[(idx >> 14) * 128 + ((idx >> 7) & 127)], code[(idx >> 14) * 128 + (idx & 127)]], -1)
    else:
        W = code[idx.clamp(max=code.shape[0] - 1)]
    W = W * lin.S_group.double().repeat_interleave(qb // 8, 0)[:, :, None]
    W[idx == 65535] = lin.O_vals.double()
    W = (W * lin.h.double()[None, :, None]).permute(0, 2, 1).reshape(out, inn)
    for size in (30.0, 1.0, 1e-2, 1e-3, 1e-4):
        x = (size * torch.randn((1, inn), generator=gen, device=DEV)).half()
        sums = (x.double() @ W.T)[0]
        groups = sums.view(-1, qb)
        lin.g = torch.exp2(-torch.log2(groups.abs().amax(1)).ceil()).clamp(2.0 ** -14, 32768.0).repeat_interleave(qb).half()
        lin.bias = None
        before = _lib.load().eptq_kernel_launch_count(1)
        # other rows of other sizes beside it must not matter
        first = lin(torch.cat([x, 100 * x.clamp(-600, 600), x * 0.01]))[0]
        lin.bias = -first
        both = first.double() + lin(x)[0].double()
        assert _lib.load().eptq_kernel_launch_count(1) - before == 2                # the multi-row kernel took both
        want = sums * lin.g.double()
        rms = want.view(-1, qb).pow(2).mean(1).sqrt().repeat_interleave(qb)
        # fp32 sums of 6176 products: below 1e-6 of a group's rms; the second result is fp16 of a difference below 2^-11
        assert float(((both - want).abs() / (rms + want.abs())).max()) <= 4e-6


@pytest.mark.parametrize("kind", ["e8_d4", "e8_lattice"])
@pytest.mark.parametrize("batch", [1, 4, 6])
def test_group_scales_infinities(kind, batch):
    """An infinity or a NaN in the activations gives what the SIMT kernel gives, also where the column is a critical block
    of some rows or a codeword coordinate is zero; rows without one are not touched."""
    import ctypes as C
    out, inn = 4096, 6176
    qd = make_layer(out, inn, seed=6, outlier_frac=0.004, bias=True, qb_size=128)
    lin = EPTQLinear.from_quantized_data(qd, torch.from_numpy(TABLES[kind]), kind).to(DEV)
    lib = _lib.load()
    col = int(lin.O_col[int(lin.O_row_ptr[40])])                         # a critical block of Q row 40
    for places in ([(0, 17, float("inf"))], [(0, col, -float("inf"))], [(batch - 1, 5, float("inf")), (batch - 1, 6000, float("inf"))],
                   [(batch // 2, col, float("nan"))], [(0, 1, float("inf")), (0, 2, -float("inf"))]):
        x = make_activations(batch, inn, seed=3).to(DEV)
        clean = lin(x)
        for b, c, v in places:
            x[b, c] = v
        before = lib.eptq_kernel_launch_count(1)
        y = lin(x)
        assert lib.eptq_kernel_launch_count(1) - before == (batch + 3) // 4
        d = lin.descriptor()
        d.h_absmax = 0.0                                                 # no bound: the SIMT kernel
        ws = torch.zeros(lib.eptq_layer_workspace_bytes(C.byref(d), batch), dtype=torch.uint8, device=DEV)
        ref = torch.empty_like(y)
        assert lib.eptq_linear_forward(C.byref(d), x.data_ptr(), ref.data_ptr(), batch, ws.data_ptr(), ws.numel(),
                                       torch.cuda.current_stream().cuda_stream) == 0
        assert torch.equal(y.isnan(), ref.isnan()) and torch.equal(y.isposinf(), ref.isposinf()) and torch.equal(y.isneginf(), ref.isneginf())
        hit = {b for b, _, _ in places}
        for b in range(batch):
            assert bool(y[b].isfinite().all()) != (b in hit)
            if b not in hit:
                assert torch.equal(y[b], clean[b])


@pytest.mark.parametrize("out,inn,batch,rows", [
    (4096, 4096, 1, False), (4096, 4096, 3, True), (4096, 4096, 8, True), (4096, 4096, 9, False), (2048, 8192, 4, True),
    (1024, 16384, 4, False), (2304, 10944, 1, True), (2304, 10880, 1, False), (1024, 4096, 16, False)])
def test_group_scales_route_by_size(out, inn, batch, rows):
    """Each side of the lines between the multi-row and the SIMT kernel, against 64 bits."""
    qd = make_layer(out, inn, seed=2, outlier_frac=0.002, qb_size=128, device=DEV)
    qd.g.mul_(inn ** -0.5)
    lin = EPTQLinear.from_quantized_data(qd, torch.from_numpy(TABLES["e8_d4"]).to(DEV), "e8_d4")
    x = make_activations(batch, inn, seed=1, device=DEV)
    lib = _lib.load()
    lin(x)
    before = [lib.eptq_kernel_launch_count(k) for k in range(6)]
    y = lin(x)
    took = [lib.eptq_kernel_launch_count(k) - b for k, b in enumerate(before)]
    assert took == ([0, (batch + 3) // 4, 0, 0, 0, 0] if rows else [0, 0, 0, 1, 0, 0])
    ref = x.double() @ lin.dequantize().double().T
    assert float((y.double() - ref).abs().max() / ref.abs().max()) <= util.REL_TOL
