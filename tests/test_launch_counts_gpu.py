"""Kernels that a composite call launches, counted as the nodes of its CUDA graph."""
import ctypes as C

import pytest

pytestmark = pytest.mark.gpu


def _launches(call):
    """Nodes of the graph of call(stream)."""
    import torch
    call(None)
    torch.cuda.synchronize()
    g, s = torch.cuda.CUDAGraph(keep_graph=True), torch.cuda.Stream()
    with torch.cuda.graph(g, stream=s):
        call(s)
    count = C.CDLL("libcudart.so.12").cudaGraphGetNodes
    count.argtypes = [C.c_void_p, C.c_void_p, C.POINTER(C.c_size_t)]
    n = C.c_size_t()
    assert count(g.raw_cuda_graph(), None, C.byref(n)) == 0
    g.instantiate()
    return n.value


@pytest.mark.parametrize("nphi", (8192, 16384))
def test_single_multiplication_scatters_its_results_in_one_launch(gpu, nphi):
    """k residues stay below the tensor cores' line and the three results' 3 k cross it at k 22."""
    import torch
    from cupoly_b200.engine import Engine, QBase
    counts = []
    for k in (21, 22):
        e = Engine(k, 0, nphi, 256)
        ins = [torch.randint(0, 1 << 62, (1, k, nphi // 2, 2), device="cuda", dtype=torch.int64) for _ in range(4)]
        outs = [e.empty(QBase) for _ in range(3)]
        e.workspace()
        counts.append(_launches(lambda s: e.bfv_mul(*outs, *ins, stream=s)))
        want = e.empty(QBase, 3)
        e.bfv_mul_batch(want, *ins, 1, e.bfv_mul_batch_workspace(1))
        assert all(torch.equal(outs[v][0], want[v]) for v in range(3))
    assert counts[0] == counts[1], counts


@pytest.mark.parametrize("nphi,k,P", [(4096, 2, 2), (4096, 2, 15), (4096, 2, 64), (8192, 5, 32), (16384, 3, 2),
                                      (16384, 3, 8), (32768, 2, 3)])
def test_the_batched_chain_launches_what_it_says(gpu, nphi, k, P):
    import torch
    from cupoly_b200.engine import Engine, QBase
    e = Engine(k, 0, nphi, 256)
    ins = [torch.randint(0, 1 << 62, (P, k, nphi // 2, 2), device="cuda", dtype=torch.int64) for _ in range(4)]
    c, ws = e.empty(QBase, 3 * P), e.bfv_mul_batch_workspace(P)
    assert _launches(lambda s: e.bfv_mul_batch(c, *ins, P, ws, stream=s)) == e.bfv_mul_batch_launches(P)


@pytest.mark.parametrize("copies", (1, 20, 300))
def test_a_mixed_batch_launches_what_it_says(gpu, copies):
    """nphi 2048 and 16384, whose transforms take one kernel each on either kind of core."""
    from cupoly_b200.batch import MixedPolymul
    mp = MixedPolymul([(2048, 4), (16384, 8)] * copies, kmax=8)
    for g in mp.groups.values():
        g["engine"].set_plan(3, 13)
        g["engine"].set_narrow_plan(0, 0, 0)
        g["engine"].set_tensor(1)
    want = sum(3 + (g["rows"] > {2048: 1150, 16384: 74}[n]) for n, g in mp.groups.items())
    assert mp.launches_per_run() == want

    def run(s):
        for g in mp.groups.values():
            mp._launch_group(g, s)

    assert _launches(run) == want
