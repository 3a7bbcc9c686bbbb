"""A training step whose gradients of weights run on a side stream gives, bit for
bit, what it gives on one stream: eagerly, on a stream of the caller's, and from a
captured graph, over repeated steps without a synchronisation between them."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("layers,batch", [(1, 64), (4, 128)])
def test_side_stream_matches_one_stream(gpu_lib, layers, batch):
    import torch
    from csrst_b200 import surrogate
    g = torch.Generator().manual_seed(batch)
    X = torch.randn(batch, 256, 64, generator=g).to(torch.bfloat16).cuda()
    T = torch.randn(batch, 256, 32, generator=g).cuda()

    def steps(net, n):
        for _ in range(n):
            net.loss_and_grad(X, T)
            net.adam()

    def run(how):
        net = surrogate.FNO(layers=layers, seed=7)
        steps(net, 1)                                # buffers exist before anything is captured
        if how == "one":
            one = net._net
            net._net = lambda *a: [n := one(*a), setattr(n, "side", None)][0]
        torch.cuda.synchronize()
        if how == "stream":
            with torch.cuda.stream(torch.cuda.Stream()):
                steps(net, 12)
        elif how == "graph":
            graph = torch.cuda.CUDAGraph()
            with torch.cuda.graph(graph):
                steps(net, 2)
            for _ in range(6):
                graph.replay()
        else:
            steps(net, 12)
        torch.cuda.synchronize()
        net.check()
        return net.w.clone(), net.g.clone(), net._bufs[(batch, True)].loss.clone()

    ref = run("one")
    assert bool(torch.isfinite(ref[0]).all()) and bool((ref[1] != 0).any())
    for how in ("two", "stream", "graph"):
        for a, b in zip(run(how), ref):
            assert torch.equal(a, b), how


def test_copies_of_a_trained_network(gpu_lib):
    import copy
    import pickle

    import torch
    from csrst_b200 import surrogate
    net = surrogate.FNO(layers=1, seed=3)
    X = torch.randn(64, 256, 64, generator=torch.Generator().manual_seed(1)).to(torch.bfloat16).cuda()
    T = torch.zeros(64, 256, 32, device="cuda")
    net.loss_and_grad(X, T)
    for other in (copy.deepcopy(net), pickle.loads(pickle.dumps(net))):
        other.loss_and_grad(X, T)
        assert torch.equal(other.g, net.g)
