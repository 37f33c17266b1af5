"""Tensor-core GEMM over K ranges, its index ring and its look-ahead for critical blocks, against the oracle."""
import numpy as np
import pytest
import torch

import oracle
from eptq_b200 import _lib
from eptq_b200.kernels.linear import EPTQLinear
from eptq_b200.synthetic import make_activations, make_layer
from tests import util

pytestmark = pytest.mark.gpu
DEV = "cuda"
TABLES = {"e8_d4": oracle.d4_table(1.75), "e8_lattice": oracle.e8_table(1.6)}


@pytest.mark.parametrize("kind", ["e8_d4", "e8_lattice"])
@pytest.mark.parametrize("out,inn,tokens,qb,frac", [
    (1024, 4096, 17, 0, 0.004),          # many ranges, a mostly empty token tile
    (264, 1096, 129, 0, 0.02),           # ragged rows, a last chunk of 8 columns
    (128, 64, 33, 0, 0.3),               # one chunk, one range
    (1024, 2056, 300, 128, 0.004),       # group scales shared by a tile
    (1024, 2056, 100, 64, 0.02),         # group scales that change inside a tile
    (136, 520, 513, 0, 1.1),             # nothing but critical blocks, reconstructed once
    (136, 520, 512, 0, 1.1),             # the same tile by tile
    (768, 768, 512, 0, 0.004),           # short rows at many tokens: one range
])
def test_ranges_match_oracle(kind, out, inn, tokens, qb, frac):
    qd = make_layer(out, inn, seed=out + inn + tokens, outlier_frac=frac, bias=(tokens % 2 == 1), qb_size=qb or None)
    lin = EPTQLinear.from_quantized_data(qd, torch.from_numpy(TABLES[kind]), kind).to(DEV)
    x = make_activations(tokens, inn, seed=tokens)
    W16 = oracle.dequantize_layer(util.qld_arrays(qd), TABLES[kind])
    ref = oracle.linear_reference(x.numpy(), W16, None if qd.bias is None else qd.bias.numpy())
    xd = x.to(DEV)
    y = lin(xd)
    assert util.max_rel_err(y.float().cpu().numpy(), ref) <= util.REL_TOL
    assert torch.equal(lin(xd), y)                       # ranges are added in a fixed order, the scratch is left clean
    W = lin.dequantize()
    assert np.array_equal(W.cpu().numpy().view(np.uint16), np.asarray(W16).view(np.uint16))     # bit-exact


@pytest.mark.parametrize("kind", ["e8_d4", "e8_lattice"])
@pytest.mark.parametrize("tokens", [100, 200, 400])
@pytest.mark.parametrize("one_range", [False, True])
def test_every_column_meets_its_own_weight(kind, tokens, one_range):
    """One-hot rows read the weights the GEMM multiplied by: a column of W16 each, exactly.  Blocks with many chunks, so
    that the index ring is refilled while the slowest warp still reads it; cold and warm L2."""
    import ctypes as C
    out = inn = 4096
    lin = EPTQLinear.from_quantized_data(make_layer(out, inn, seed=3, device=DEV), torch.from_numpy(TABLES[kind]).to(DEV), kind)
    W = lin.dequantize()
    d = lin.descriptor()
    lib = _lib.load()
    need = 1 << 20 if one_range else lib.eptq_layer_workspace_bytes(C.byref(d), tokens)
    ws = torch.zeros(need, dtype=torch.uint8, device=DEV)
    flush = torch.empty(1 << 28, dtype=torch.uint8, device=DEV)
    rows = torch.arange(tokens, device=DEV)
    for rep in range(16):
        cols = (rows * inn // tokens + 5 * rep) % inn
        x = torch.zeros((tokens, inn), dtype=torch.float16, device=DEV)
        x[rows, cols] = 1
        if rep % 2 == 0:
            flush.zero_()
        y = torch.empty((tokens, out), dtype=torch.float16, device=DEV)
        st = lib.eptq_linear_forward(C.byref(d), x.data_ptr(), y.data_ptr(), tokens, ws.data_ptr(), ws.numel(),
                                     torch.cuda.current_stream().cuda_stream)
        assert st == 0 and torch.equal(y, W[:, cols].T)


@pytest.mark.parametrize("kind", ["e8_d4", "e8_lattice"])
def test_ranges_over_token_tiles(kind):
    """Scratch that holds the partial sums but not the weight: tile by tile, K ranges, more than one token tile."""
    import ctypes as C
    out, inn, tokens = 1024, 32768, 700
    lin = EPTQLinear.from_quantized_data(make_layer(out, inn, seed=8, device=DEV), torch.from_numpy(TABLES[kind]).to(DEV), kind)
    d = lin.descriptor()
    lib = _lib.load()
    x = make_activations(tokens, inn, seed=9, device=DEV)
    ref = x.double() @ lin.dequantize().double().T
    ws = torch.zeros((1 << 20) + (64 << 20), dtype=torch.uint8, device=DEV)          # the weight alone is 64 MiB
    ws = ws[: ws.numel() - 256]
    before = [lib.eptq_kernel_launch_count(k) for k in range(6)]
    ys = []
    for _ in range(3):
        y = torch.empty((tokens, out), dtype=torch.float16, device=DEV)
        assert lib.eptq_linear_forward(C.byref(d), x.data_ptr(), y.data_ptr(), tokens, ws.data_ptr(), ws.numel(),
                                       torch.cuda.current_stream().cuda_stream) == 0
        ys.append(y)
    assert [lib.eptq_kernel_launch_count(k) - b for k, b in enumerate(before)] == [0, 0, 0, 0, 3, 0]     # no reconstruction
    assert float((ys[0].double() - ref).abs().max() / ref.abs().max()) <= util.REL_TOL
    assert torch.equal(ys[0], ys[1]) and torch.equal(ys[0], ys[2])
    assert int(ws[:4096].view(torch.int32).abs().max()) == 0                         # counters left at zero, no time-out
