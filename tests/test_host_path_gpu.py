"""The native host path of single packed products (csrc/host_path.cpp) against the Python path it stands in for: the same
bits where it takes a call, None - so that the Python path serves or refuses the call - everywhere else."""
import pytest
import torch

from bitmtp_b200 import model as BM
from bitmtp_b200 import native, ops, synthetic
from bitmtp_b200.model import T2LinearKernel

pytestmark = pytest.mark.gpu
DEV = torch.device("cuda:0")


def _operands(rows, n=264, k=768, seed=0):
    gen = torch.Generator(device=DEV).manual_seed(seed)
    packed, scale = synthetic.device_ternary(n, k, gen, DEV)
    x = torch.randn(rows, k, generator=gen, device=DEV).to(torch.bfloat16)
    native.lib()
    return x, packed, scale


def _without_host(monkeypatch, fn):
    with monkeypatch.context() as m:
        m.setattr(native, "_host", None)
        return fn()


@pytest.mark.parametrize("shape", [(1,), (17,), (32,), (1, 1), (2, 5)])
def test_operator(monkeypatch, shape):
    rows = shape[0] * (shape[1] if len(shape) == 2 else 1)
    x, packed, scale = _operands(rows)
    q, s = ops.quant_rows(x)
    q, s = q.view(*shape, -1), s.view(*shape, 1)
    got = native._host.linear(q, packed, s, scale)
    want = _without_host(monkeypatch, lambda: BM.t2g128_int8xint2_linear(q, packed, s, scale))
    assert got.shape == want.shape and got.dtype == want.dtype and torch.equal(got.view(torch.int16), want.view(torch.int16))
    with torch.inference_mode():
        assert BM.t2g128_int8xint2_linear(q, packed, s, scale).is_inference()


@pytest.mark.parametrize("rows", [1, 2, 9, 16, 17, 32, 33, 200])
@pytest.mark.parametrize("n,k", [(264, 768), (8, 128), (4104, 1024), (520, 384), (2048, 6144)])
def test_module(monkeypatch, rows, n, k):
    x, packed, scale = _operands(rows, n, k, seed=rows)
    layer = T2LinearKernel(k, n).to(DEV)
    layer.weight.data, layer.weight_scale = packed, scale
    for xs in (x, x.view(1, rows, k), x[0]):
        got = native._host.linear_rows(xs, layer.weight.data, scale, ops.gemv_serves_rows, ops.GEMM_WIDE_MAX_ROWS)
        want = _without_host(monkeypatch, lambda: layer(xs))
        assert got.shape == want.shape and torch.equal(got.view(torch.int16), want.view(torch.int16))
        assert torch.equal(layer(xs).view(torch.int16), want.view(torch.int16))
    # every second column: not contiguous, served by the Python path after a copy
    wide = torch.stack([x, x], dim=-1)[..., 0]
    assert native._host.linear_rows(wide, packed, scale, ops.gemv_serves_rows, ops.GEMM_WIDE_MAX_ROWS) is None
    assert torch.equal(layer(wide).view(torch.int16), layer(x).view(torch.int16))


class _Tagged(torch.Tensor):
    pass


def test_what_is_left_to_the_python_path():
    x, packed, scale = _operands(4)
    q, s = ops.quant_rows(x)
    bad = [(q.cpu(), packed, s, scale), (q[:, :640], packed, s, scale), (q, packed.t(), s, scale),
           (q, packed, s, scale[:, :2]), (q.float(), packed, s, scale), (q, packed, s.double(), scale),
           (q, packed, s, scale.float()), (q, packed, s[:3], scale), (q, packed, s.view(1, 4), scale), (q, packed, None, scale),
           (q[None, None], packed, s, scale), (q.as_subclass(_Tagged), packed, s, scale), (q[:0], packed, s[:0], scale),
           (q, packed[:12], s, scale[:12]), (q.repeat(9, 1), packed, s.repeat(9, 1), scale)]
    for args in bad:
        assert native._host.linear(*args) is None
    for args in (bad[0], bad[1], bad[3], bad[5], bad[13], bad[14]):
        with pytest.raises((RuntimeError, ValueError)):
            BM.t2g128_int8xint2_linear(*args)
    with pytest.raises(RuntimeError):                       # the registry does not list these sizes
        BM.t2g128_int8xint2_linear(q, packed, s, scale, validate_registry=True)

    class Mode(torch.overrides.TorchFunctionMode):
        def __torch_function__(self, func, types, args=(), kwargs=None):
            return func(*args, **(kwargs or {}))

    with Mode():
        assert native._host.linear(q, packed, s, scale) is None

    def inside(row):
        assert native._host.linear_rows(row, packed, scale, ops.gemv_serves_rows, ops.GEMM_WIDE_MAX_ROWS) is None
        return row

    torch.func.vmap(inside)(x.view(2, 2, -1))
    torch.func.jvp(inside, (x,), (x,))
    assert native._host.linear_rows(x.float(), packed, scale, ops.gemv_serves_rows, ops.GEMM_WIDE_MAX_ROWS) is None
    shifted = torch.cat([scale.view(-1)[:4], scale.view(-1)])[4:].view_as(scale)
    assert native._host.linear_rows(x, packed, shifted, ops.gemv_serves_rows, ops.GEMM_WIDE_MAX_ROWS) is None


def _shifted(t, elements):
    """The same values, contiguous, off a 16-byte boundary."""
    return torch.cat([t.reshape(-1)[:elements], t.reshape(-1)])[elements:].view_as(t)


@pytest.mark.parametrize("host", [True, False])
def test_a_call_that_the_library_refuses_raises(monkeypatch, host):
    """Operands off a 16-byte boundary, and rows too long for the shared memory of the lanes-across-K kernel: an error and no
    tensor of whatever memory held, by the native host path and by the Python path behind it."""
    x, packed, scale = _operands(4)
    q, s = ops.quant_rows(x)
    long_x, long_packed, long_scale = _operands(16, 8, 16512)
    long_q, long_s = ops.quant_rows(long_x)
    if not host:
        monkeypatch.setattr(native, "_host", None)
    for args in ((_shifted(q, 8), packed, s, scale), (q, _shifted(packed, 8), s, scale), (q, packed, s, _shifted(scale, 4)),
                 (long_q, long_packed, long_s, long_scale)):
        assert all(t.is_contiguous() for t in args)
        with pytest.raises(native.NativeError):
            BM.t2g128_int8xint2_linear(*args)
    torch.cuda.synchronize()
    got = BM.t2g128_int8xint2_linear(q, packed, _shifted(s, 1), scale)       # multipliers need no more than their own size
    assert torch.equal(got, BM.t2g128_int8xint2_linear(q, packed, s, scale))


def test_nested_tensors_are_left_to_the_python_path():
    """Strided nested tensors are exact torch.Tensor objects on a CUDA device, but asking them for a ragged size throws."""
    x, packed, scale = _operands(4)
    q, s = ops.quant_rows(x)
    for widths in ((768, 768), (768, 640)):
        nq, ns, nx = (torch.nested.nested_tensor([t[:2, :w], t[2:, :w]], layout=torch.strided)
                      for t, w in ((q, widths[1]), (s, 1), (x, widths[1])))
        ragged = torch.nested.nested_tensor([q[:3, :widths[0]], q[3:, :widths[1]]], layout=torch.strided)
        assert type(ragged) is torch.Tensor and ragged.is_cuda and ragged.layout == torch.strided
        for args in ((nq, packed, s, scale), (ragged, packed, s, scale), (q, ragged, s, scale), (q, packed, ns, scale),
                     (q, packed, s, ragged)):
            assert native._host.linear(*args) is None
        for args in ((nx, packed, scale), (ragged, packed, scale), (x, ragged, scale), (x, packed, ragged)):
            assert native._host.linear_rows(*args, ops.gemv_serves_rows, ops.GEMM_WIDE_MAX_ROWS) is None
        with pytest.raises(RuntimeError):
            BM.t2g128_int8xint2_linear(ragged, packed, s, scale)


@pytest.mark.parametrize("host", [True, False])
def test_running_out_of_memory_is_torchs_own_error(monkeypatch, host):
    """A product whose output (256 GiB) fits no device: torch.OutOfMemoryError, which callers catch to retry with less."""
    n, rows = 1 << 22, 1 << 15
    layer = T2LinearKernel(128, 8).to(DEV)
    layer.weight.data = torch.zeros(n, 32, dtype=torch.int8, device=DEV)
    layer.weight_scale = torch.zeros(n, 1, dtype=torch.bfloat16, device=DEV)
    layer.out_features = n
    native.lib()
    if not host:
        monkeypatch.setattr(native, "_host", None)
    with pytest.raises(torch.OutOfMemoryError):
        layer(torch.zeros(rows, 128, dtype=torch.bfloat16, device=DEV))


def test_the_drop_in_symbol():
    """The C symbol that programs written for the reference bind: the operator's bits, and nothing written on refusal."""
    x, packed, scale = _operands(9)
    q, s = ops.quant_rows(x)
    out = torch.full((9, 264), 7.0, dtype=torch.bfloat16, device=DEV)
    call = native.lib().t2g128_int8xint2_linear
    stream = torch.cuda.current_stream().cuda_stream
    call(q.data_ptr() + 8, packed.data_ptr(), out.data_ptr(), s.data_ptr(), scale.data_ptr(), 9, 264, 768, stream)
    torch.cuda.synchronize()
    assert bool((out == 7.0).all())
    call(q.data_ptr(), packed.data_ptr(), out.data_ptr(), s.data_ptr(), scale.data_ptr(), 9, 264, 768, stream)
    want = BM.t2g128_int8xint2_linear(q, packed, s, scale)
    torch.cuda.synchronize()
    assert torch.equal(out.view(torch.int16), want.view(torch.int16))


def test_the_operators_output_is_an_ordinary_tensor(monkeypatch):
    """What the host path allocates is what torch.empty gives in each setting: shape, strides, type, device, inference tensor or
    not, in a memory pool of its own under capture, and the same bits where uninitialised memory is filled."""
    x, packed, scale = _operands(6)
    q, s = ops.quant_rows(x)
    want = _without_host(monkeypatch, lambda: BM.t2g128_int8xint2_linear(q, packed, s, scale))
    for inference in (False, True):
        with torch.inference_mode(inference):
            for view in ((6,), (2, 3)):
                got = native._host.linear(q.view(*view, -1), packed, s.view(*view, 1), scale)
                ref = torch.empty((*view, 264), dtype=torch.bfloat16, device=DEV)
                for name in ("shape", "dtype", "device", "layout", "requires_grad"):
                    assert getattr(got, name) == getattr(ref, name), name
                assert got.stride() == ref.stride() and got.is_inference() == ref.is_inference() == inference
                assert torch.equal(got.view(6, -1).view(torch.int16), want.view(torch.int16))
    torch.use_deterministic_algorithms(True)
    try:
        assert torch.equal(native._host.linear(q, packed, s, scale).view(torch.int16), want.view(torch.int16))
    finally:
        torch.use_deterministic_algorithms(False)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        out = BM.t2g128_int8xint2_linear(q, packed, s, scale)
    out.zero_()
    graph.replay()
    torch.cuda.synchronize()
    assert torch.equal(out.view(torch.int16), want.view(torch.int16))
    traced = torch.jit.trace(lambda a: BM.t2g128_int8xint2_linear(a, packed, s, scale), (q,), check_trace=False)
    assert traced(q).shape == want.shape
