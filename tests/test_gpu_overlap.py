"""Kernels of one native call that start while their predecessor drains: who may, and that results do not depend on it."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture(autouse=True)
def restore_budget():
    from bamboo_b200 import lib
    lib.load()
    yield
    lib.GEMM_MAX_CTAS = 0


def _arena(mods):
    from bamboo_b200.arena import ParamArena
    return ParamArena([p for m in mods for p in m.parameters()], torch.device("cuda"), torch.bfloat16)


def _block(heads, head_dim):
    from bamboo_b200 import layers
    torch.manual_seed(3)
    return layers.TransformerBlock(heads * head_dim, heads, 4 * heads * head_dim, causal=True)


def _conv(cin, cout, k, stride=1):
    from bamboo_b200 import resnet
    return resnet.ConvBN(cin, cout, k, stride=stride, relu=True, generator=torch.Generator().manual_seed(3))


def captured(fn):
    """The call as a graph that is not run (its caches and attributes are set up by a call before)."""
    from cuda.bindings import runtime as rt
    fn()
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph(keep_graph=True)
    with torch.cuda.graph(graph):
        fn()
    return graph, rt.cudaGraph_t(graph.raw_cuda_graph()), rt


def _programmatic_edges(fn):
    """Edges of the captured call along which a kernel may start before the one in front of it has ended."""
    graph, handle, rt = captured(fn)
    err, *_, n = rt.cudaGraphGetEdges_v2(handle)
    assert err == rt.cudaError_t.cudaSuccess
    err, _from, _to, data, n = rt.cudaGraphGetEdges_v2(handle, n)
    assert err == rt.cudaError_t.cudaSuccess and n > 0
    return sum(int(d.type) == int(rt.cudaGraphDependencyType.cudaGraphDependencyTypeProgrammatic) for d in data[:n])


def kernel_nodes(handle, rt):
    err, _nodes, n = rt.cudaGraphGetNodes(handle)
    err, nodes, n = rt.cudaGraphGetNodes(handle, n)
    assert err == rt.cudaError_t.cudaSuccess
    return [v for v in nodes[:n] if rt.cudaGraphNodeGetType(v)[1] == rt.cudaGraphNodeType.cudaGraphNodeTypeKernel]


@pytest.mark.parametrize("layer", ["block", "conv"])
@pytest.mark.parametrize("budget,overlaps", [(0, True), (-1, False), (20, False)])
def test_work_beside_the_main_stream_is_launched_plainly(layer, budget, overlaps):
    """Redundant work - short CTAs (-1) or a budget of CTAs - must hand its SMs back: a kernel that waits keeps its SMs."""
    from bamboo_b200 import lib
    m = _block(4, 64) if layer == "block" else _conv(64, 64, 3)
    _arena([m])
    x = torch.randn(*((2, 100, 256) if layer == "block" else (4, 14, 14, 64)), device="cuda").bfloat16()

    def fn():
        with torch.no_grad():
            m(x)
    lib.GEMM_MAX_CTAS = budget
    edges = _programmatic_edges(fn)
    assert edges > 0 if overlaps else edges == 0


# (a reduction of fewer than sixteen k-blocks is not split and a single key tile adds to dQ once: every sum has one order)
@pytest.mark.parametrize("heads,head_dim,batch,seq", [(4, 64, 2, 100), (2, 128, 3, 70), (16, 64, 1, 128)])
def test_a_block_gives_the_same_bits_with_and_without_overlap(heads, head_dim, batch, seq):
    from bamboo_b200 import layers, lib
    m = _block(heads, head_dim)
    arena = _arena([m])
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    g = torch.Generator(device="cuda").manual_seed(4)
    x = torch.randn(batch, seq, heads * head_dim, device="cuda", generator=g).bfloat16()
    dout = torch.randn(batch, seq, heads * head_dim, device="cuda", generator=g).bfloat16()

    def step(budget):
        lib.GEMM_MAX_CTAS = budget
        arena.grad.zero_()
        xi = x.clone().requires_grad_(True)
        y = m(xi)
        y.backward(dout)
        layers.wgrad_sync(x.device)
        return y.detach(), xi.grad, arena.grad.clone()
    want = step(sms)                            # the same grids, launched plainly
    for _ in range(20):
        for a, b in zip(step(0), want):
            assert torch.equal(a, b)
    assert lib.read_status() == 0


@pytest.mark.parametrize("cin,cout,k,stride", [(64, 64, 3, 1), (64, 128, 3, 2), (16, 64, 1, 1), (8, 32, 7, 2)])
def test_a_convolution_gives_the_same_bits_with_and_without_overlap(cin, cout, k, stride):
    from bamboo_b200 import lib, resnet
    m = resnet.ConvBN(cin, cout, k, stride=stride, relu=True, generator=torch.Generator().manual_seed(3))
    arena = _arena([m])
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    g = torch.Generator(device="cuda").manual_seed(4)
    x = torch.randn(3, 15, 15, cin, device="cuda", generator=g).bfloat16()

    def step(budget):
        lib.GEMM_MAX_CTAS = budget
        arena.grad.zero_()
        xi = x.clone().requires_grad_(True)
        y = m(xi)
        y.backward(y.detach() - 0.5)
        return y.detach(), xi.grad, arena.grad.clone()
    want = step(sms)
    for _ in range(20):
        for a, b in zip(step(0), want):
            assert torch.equal(a, b)
    assert lib.read_status() == 0


@pytest.mark.parametrize("make,shape", [(lambda: _block(4, 64), (2, 100, 256)), (lambda: _block(2, 128), (3, 70, 256)),
                                        (lambda: _conv(64, 64, 3), (3, 15, 15, 64)), (lambda: _conv(64, 64, 3, 2), (3, 15, 15, 64)),
                                        (lambda: _conv(16, 64, 1), (3, 15, 15, 16)), (lambda: _conv(64, 16, 3), (3, 15, 15, 64)),
                                        (lambda: _conv(8, 32, 7, 2), (3, 15, 15, 8))])
def test_launch_accounting_is_that_of_the_captured_call(make, shape):
    """lib.LAUNCHES grows by the kernels that a layer's forward and backward call launch, on whichever route."""
    from bamboo_b200 import layers, lib
    m = make()
    _arena([m])
    x = torch.randn(*shape, device="cuda").bfloat16().requires_grad_(True)
    dout, counted = torch.ones_like(m(x)), []

    def fn():
        before = lib.LAUNCHES
        torch.autograd.grad(m(x), x, dout)
        if isinstance(m, layers.TransformerBlock):
            layers.wgrad_sync(x.device)              # (a convolution layer has no work on that stream to join)
        counted.append(lib.LAUNCHES - before)
    graph, handle, rt = captured(fn)
    nodes = len(kernel_nodes(handle, rt))
    assert counted == [nodes, nodes]
