"""The tensor-core kernels with two streams in flight: their blocks then share the SMs, start at any
time and in any order, and the results are those of one stream.  Every launch is above the tensor
cores' line, at the two block sizes whose passes have four tiles or two that exchange halves, and
with the split stage."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nphi,k,P", [(8192, 5, 47), (16384, 4, 33), (32768, 4, 9)])
def test_two_streams_equal_one(gpu, nphi, k, P):
    import torch
    from cupoly_b200.engine import FORWARD, INVERSE, Engine, QBase
    rounds, N = 6, nphi // 2
    e, o = Engine(k, 0, nphi, 256), Engine(k, 0, nphi, 256)
    o.set_tensor(0)
    assert e.dgt_launches(P * k)[1] and not o.dgt_launches(4 * P * k)[1]
    g = torch.Generator(device="cuda").manual_seed(nphi)

    def rand(*shape):
        return torch.randint(0, 1 << 62, shape, generator=g, device="cuda", dtype=torch.int64)

    lanes = []
    for i in range(2):
        lane = {"s": torch.cuda.Stream(), "x": [rand(P, k, N, 2) for _ in range(rounds)],
                "ins": [rand(P, k, N, 2) for _ in range(4)], "coefs": rand(P, nphi, k)}
        lane["coefs"][..., k - 1] >>= k  # below the product of the primes
        lane["y"] = [x.clone() for x in lane["x"]]
        lane["c"] = [e.empty(QBase, 3 * P) for _ in range(rounds)]
        lane["res"] = [e.empty(QBase, P) for _ in range(rounds)]
        lane["back"] = [torch.empty_like(lane["coefs"]) for _ in range(rounds)]
        lane["ws"] = e.bfv_mul_batch_workspace(P)
        lanes.append(lane)
    torch.cuda.synchronize()
    for r in range(rounds):
        for i, lane in enumerate(lanes):
            s = lane["s"]
            steps = [lambda: e.dgt(lane["y"][r], QBase, FORWARD, P, stream=s),
                     lambda: e.bfv_mul_batch(lane["c"][r], *lane["ins"], P, lane["ws"], stream=s),
                     lambda: (e.crt(lane["res"][r], lane["coefs"], QBase, stream=s),
                              e.icrt(lane["back"][r], lane["res"][r], QBase, stream=s))]
            for v in range(3):  # the two streams are at different kernels
                steps[(v + i) % 3]()
            e.dgt(lane["y"][r], QBase, INVERSE, P, stream=s)
            e.dgt(lane["y"][r], QBase, FORWARD, P, stream=s)
    torch.cuda.synchronize()
    e.check()
    for lane in lanes:
        want = e.empty(QBase, 3 * P)
        o.bfv_mul_batch(want, *lane["ins"], P, lane["ws"])
        res = e.empty(QBase, P)
        for q in range(P):  # single polynomials: below the tensor cores' line for I/O
            o.crt(res[q:q + 1], lane["coefs"][q:q + 1], QBase)
        for r in range(rounds):
            f = lane["x"][r].clone()
            o.dgt(f, QBase, FORWARD, P)
            assert torch.equal(lane["y"][r], f), r
            assert torch.equal(lane["c"][r], want), r
            assert torch.equal(lane["res"][r], res), r
            assert torch.equal(lane["back"][r], lane["coefs"]), r
