"""The native host path of module calls: it follows the module it was made for."""
import pytest
import torch

import oracle
from eptq_b200.kernels.linear import EPTQLinear, forward_group
from eptq_b200.synthetic import make_activations, make_layer

pytestmark = pytest.mark.gpu
DEV = "cuda"
_tables: dict = {}


def table(kind):
    """One codebook tensor: layers of a group share it."""
    if kind not in _tables:
        _tables[kind] = torch.from_numpy(oracle.d4_table(1.75) if kind == "e8_d4" else oracle.e8_table(1.6)).to(DEV)
    return _tables[kind]


def layer(kind, out=1024, inn=2048, seed=1, **kw):
    qd = make_layer(out, inn, seed=seed, device=DEV, outlier_frac=0.01, **kw)
    return EPTQLinear.from_quantized_data(qd, table(kind), kind)


def fresh(lin):
    """A new module over the present buffers."""
    return EPTQLinear(lin.Q, lin._codebook, lin.g, lin.h, lin.O_vals, lin.O_col, lin.O_row_ptr, lin.bias, lin.quantizer_type,
                      S_group=lin.S_group, codebook32=lin._codebook32)


@pytest.mark.parametrize("kind", ["e8_d4", "e8_lattice"])
@pytest.mark.parametrize("tokens", [1, 3])
def test_calls_follow_changed_buffers(kind, tokens):
    lin, other = layer(kind, bias=True), layer(kind, seed=2)
    x = make_activations(tokens, 2048, seed=9, device=DEV)
    changes = [
        lambda: setattr(lin, "bias", lin.bias * -3),
        lambda: setattr(lin, "g", lin.g * 2),
        lambda: setattr(lin, "O_vals", lin.O_vals * 4) or setattr(lin, "crit_O", fresh(lin).crit_O),
        lambda: lin.h.mul_(1000),                       # in place: x * h * 2^-e would leave fp16 with the old bound
        lambda: lin.h.div_(4000),
        lambda: setattr(lin, "bias", None),
    ]
    lin.g.mul_(2.0 ** -8)
    for change in [lambda: None, *changes]:
        change()
        ref = fresh(lin)
        assert torch.allclose(lin(x).float(), ref(x).float(), rtol=2e-3, atol=2e-3 * float(ref(x).float().abs().max()))
        a, b = forward_group([lin, other], [x, x])
        ra, rb = forward_group([ref, other], [x, x])
        assert torch.isfinite(a).all() and torch.allclose(a.float(), ra.float(), rtol=2e-3, atol=2e-3 * float(ra.float().abs().max()))
        assert torch.equal(lin.dequantize(), ref.dequantize())


@pytest.mark.parametrize("kind", ["e8_d4", "e8_lattice"])
def test_group_scales_follow_changed_buffers(kind):
    lin = layer(kind, out=4096, inn=6176, qb_size=128)
    x = make_activations(1, 6176, seed=9, device=DEV)
    lin.g.mul_(2.0 ** -12)
    for change in (lambda: None, lambda: lin.S_group.mul_(4096), lambda: setattr(lin, "S_group", lin.S_group / 512)):
        change()
        ref = fresh(lin)
        y, r = lin(x).float(), ref(x).float()
        assert torch.isfinite(y).all() and torch.allclose(y, r, rtol=2e-3, atol=2e-3 * float(r.abs().max()))
        assert torch.equal(lin.dequantize(), ref.dequantize())


def test_changed_scales_then_capture():
    """A capture cannot read the new maxima back; the call is recorded with kernels that need none."""
    lin = layer("e8_d4")
    x = make_activations(1, 2048, seed=9, device=DEV)
    side = torch.cuda.Stream()
    with torch.cuda.stream(side):
        lin(x)
        lin.h.mul_(0.5)
        side.synchronize()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=side):
            y = lin(x)
        graph.replay()
        side.synchronize()
    ref = fresh(lin)(x).float()
    assert torch.allclose(y.float(), ref, rtol=2e-3, atol=2e-3 * float(ref.abs().max()))
    assert torch.allclose(lin(x).float(), ref, rtol=2e-3, atol=2e-3 * float(ref.abs().max()))


def in_threads(jobs):
    """Run the jobs at the same time, switching between them as often as the interpreter can; errors surface."""
    import sys
    import threading
    errors = []
    start = threading.Barrier(len(jobs))

    def body(job):
        try:
            start.wait()
            job()
        except BaseException as e:                      # noqa: BLE001 - reported below
            errors.append(e)

    interval = sys.getswitchinterval()
    sys.setswitchinterval(1e-6)
    try:
        threads = [threading.Thread(target=body, args=(job,)) for job in jobs]
        for t in threads:
            t.start()
        for t in threads:
            t.join()
    finally:
        sys.setswitchinterval(interval)
    if errors:
        raise errors[0]


def test_scratch_outgrown_by_another_thread():
    """One thread's calls keep the scratch they were given while another's replace it with larger ones."""
    lin = layer("e8_d4", out=2048, inn=2048)
    small, big = make_activations(40, 2048, seed=4, device=DEV), make_activations(500, 2048, seed=5, device=DEV)
    want_small, want_big = lin(small), {t: lin(big[:t].contiguous()) for t in range(100, 501, 50)}
    for _ in range(5):
        side = torch.cuda.Stream()                      # a stream without scratch
        side.wait_stream(torch.cuda.current_stream())

        def steady():
            with torch.cuda.stream(side):
                for _ in range(200):
                    assert torch.equal(lin(small), want_small)

        def growing():
            with torch.cuda.stream(side):
                for t, want in want_big.items():
                    torch.full((1 << 20,), 255, dtype=torch.uint8, device=DEV)          # takes freed memory
                    assert torch.equal(lin(big[:t].contiguous()), want)

        in_threads([steady, growing])
    torch.cuda.synchronize()


@pytest.mark.parametrize("tokens", [600, 1100])
def test_two_threads_reconstruct_into_one_scratch(tokens):
    """Above 512 tokens a call reconstructs its weight into the stream's scratch and multiplies from there."""
    lins = [layer(kind, out=1024, inn=1024, seed=n) for n, kind in enumerate(("e8_d4", "e8_d4", "e8_lattice"))]
    x = make_activations(tokens, 1024, seed=4, device=DEV)
    decode = layer("e8_d4", out=2048, inn=2048, seed=7)                     # one launch, partial sums in the same place
    xd = make_activations(8, 2048, seed=5, device=DEV)
    want, want_d = [lin(x) for lin in lins], decode(xd)

    def repeat(lin, x, want):
        def job():
            got = [lin(x) for _ in range(150)]
            assert all(torch.equal(y, want) for y in got)
        return job

    in_threads([repeat(lin, x, w) for lin, w in zip(lins, want)] + [repeat(decode, xd, want_d)])


def test_group_inputs_of_other_shapes():
    """Inputs after the first may have any shape with as many values, attention heads not yet joined for instance."""
    a, b = layer("e8_d4"), layer("e8_d4", seed=2)
    x, z = make_activations(3, 2048, seed=9, device=DEV), make_activations(3, 2048, seed=8, device=DEV)
    ya, yb = forward_group([a, b], [x, z])
    for other in (z.view(3, 16, 128), z.view(-1), z.view(1, 3, 2048), z.view(3, 1, 2048).float()):
        oa, ob = forward_group([a, b], [x, other])
        assert torch.equal(oa, ya) and torch.equal(ob, yb.to(other.dtype)) and ob.shape == yb.shape
    with pytest.raises(RuntimeError):
        forward_group([a, b], [x, z.view(-1)[:-1]])
    with pytest.raises(RuntimeError):
        forward_group([a, b], [x, z[:2]])


def test_scratch_kept_for_graphs_is_bounded():
    """Scratch a graph was captured with outlives its replacement; what is kept stays below what is in use."""
    from eptq_b200 import _lib
    host = _lib.host()
    index = torch.cuda.current_device()
    before = {t.data_ptr() for t in host.scratch_of_device(index)}
    lin = layer("e8_d4", out=2048, inn=1024)
    side = torch.cuda.Stream()
    graphs = []
    with torch.cuda.stream(side):
        for t in range(600, 1000, 50):                  # each asks for a little more scratch than the one before
            big = layer("e8_d4", out=2 * t // 16 * 16, inn=1024, seed=t)
            x = make_activations(t, 1024, seed=t, device=DEV)
            want = big(x)
            graph = torch.cuda.CUDAGraph()
            with torch.cuda.graph(graph, stream=side):
                y = big(x)
            graphs.append((graph, big, x, y, want))
        for graph, _, _, y, want in graphs:
            y.zero_()
            graph.replay()
            assert torch.equal(y, want)
        lin(make_activations(1, 1024, seed=1, device=DEV))
        current = host.scratch(index, 1)
    sizes = [t.numel() for t in host.scratch_of_device(index) if t.data_ptr() not in before and t.data_ptr() != current.data_ptr()]
    assert sizes and sum(sizes) <= current.numel()
