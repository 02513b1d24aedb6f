"""What a captured call consists of: which kernels start as dependents of the one before them."""
import ctypes

import pytest
import torch

import engine_b200
from engine_b200 import decode

pytestmark = pytest.mark.gpu

KERNEL_NODE, PROGRAMMATIC = 0, 1   # cudaGraphNodeTypeKernel, cudaGraphDependencyTypeProgrammatic


class EdgeData(ctypes.Structure):   # cudaGraphEdgeData
    _fields_ = [("from_port", ctypes.c_ubyte), ("to_port", ctypes.c_ubyte), ("type", ctypes.c_ubyte), ("reserved", ctypes.c_ubyte * 5)]


def runtime():
    return ctypes.CDLL("libcudart.so.12")   # the one the library is linked with


def captured(stream, fn):
    """fn's launches as a graph (fn has run before: a capture must not set kernel attributes)."""
    with torch.cuda.stream(stream):
        fn()
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph(keep_graph=True)
    with torch.cuda.graph(graph, stream=stream):
        fn()
    return graph


def dependent_edges(graph):
    raw, count = ctypes.c_void_p(graph.raw_cuda_graph()), ctypes.c_size_t(64)
    ends, edges = [(ctypes.c_void_p * 64)() for _ in range(2)], (EdgeData * 64)()
    assert runtime().cudaGraphGetEdges_v2(raw, ends[0], ends[1], edges, ctypes.byref(count)) == 0
    return [edges[i].type == PROGRAMMATIC for i in range(count.value)]


@pytest.fixture(scope="module")
def own():
    context = engine_b200.RibnContext(0, torch.cuda.Stream())
    yield context
    context.close()


# a decode step of up to 64 sequences starts its operators one after the other, whatever the hidden size; a prompt chunk does not
@pytest.mark.parametrize("rows,length,dependent", [(1, 4096, False), (64, 4096, False), (64, 5120, False), (64, 8192, False), (65, 4096, True),
                                                   (65, 1024, True), (512, 5120, True)])
def test_residual_add_of_a_decode_step_is_a_plain_launch(own, rows, length, dependent):
    ops = decode.CudaDenseOps(own)
    y, x = torch.zeros(rows, length, device=own.device), torch.ones(rows, length, device=own.device)

    def twice():
        ops.residual_add(y, x)
        ops.residual_add(y, x)

    graph = captured(own.stream, twice)
    assert dependent_edges(graph) == [dependent]
    before = y.clone()
    with torch.cuda.stream(own.stream):
        graph.instantiate()
        graph.replay()
    own.synchronize()
    assert torch.equal(y, before + 2)


def kernel_nodes(graph):
    raw, count = ctypes.c_void_p(graph.raw_cuda_graph()), ctypes.c_size_t(4096)
    nodes, kind = (ctypes.c_void_p * 4096)(), ctypes.c_int()
    assert runtime().cudaGraphGetNodes(raw, nodes, ctypes.byref(count)) == 0
    found = 0
    for i in range(count.value):
        assert runtime().cudaGraphNodeGetType(ctypes.c_void_p(nodes[i]), ctypes.byref(kind)) == 0
        found += kind.value == KERNEL_NODE
    return found


# one row, shared images, paired and separate launches, the batch kernel; both geometries' row lengths
@pytest.mark.parametrize("members", [1, 2, 3, 8, 9, 33])
@pytest.mark.parametrize("hidden,intermediate", [(4096, 12288), (5120, 6400)])
def test_launches_per_step_are_the_kernels_of_the_step(own, members, hidden, intermediate):
    geometry = decode.DenseGeometry(hidden, 2, 16, 4, 128, intermediate, 2048)
    weights = decode.random_weights(own, geometry, seed=3)
    decoder = decode.CudaDenseDecode(own, geometry, weights, members, 64)
    try:
        graph = captured(own.stream, decoder._step)
        assert decoder.launches_per_step == kernel_nodes(graph)
    finally:
        own.set_option("tc_f32_activations", 0)
