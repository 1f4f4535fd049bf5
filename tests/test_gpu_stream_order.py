"""Kernels that become resident while the one ahead of them on the stream still runs: calls that reuse each other's buffers,
issued back to back and from a captured graph, must give bit for bit what they give with a synchronisation after each."""
import threading

import pytest
import torch

from siglip_b200 import synth

pytestmark = pytest.mark.gpu
DEV = "cuda"


def _chain(eng, rows, d, ff, seed):
    g = torch.Generator(device=DEV).manual_seed(seed)
    weight = lambda n, k: synth.quantize_e4m3(torch.randn((n, k), generator=g, device=DEV) * 0.05)[0]
    codes = lambda cols: torch.zeros((rows, synth.pitch128(cols)), dtype=torch.uint8, device=DEV)[:, :cols]
    one, scale = torch.ones(1, device=DEV), torch.full((1,), 0.02, device=DEV)
    wq, w1, w2 = weight(d, d), weight(ff, d), weight(d, ff)
    x0 = torch.randn((rows, d), generator=g, device=DEV).to(torch.bfloat16)
    pixels = torch.rand((1, 3, 64, 64), generator=g, device=DEV)
    x, y, a, hidden, patches = x0.clone(), torch.empty_like(x0), codes(d), codes(ff), codes(768)[:16]

    def run(step):
        """x -> two rounds of LayerNorm / projection / MLP that overwrite a, hidden, x and y while their readers may still run."""
        for buf, out in ((x, y), (y, x)):
            eng.layernorm_quantize(buf, None, None, 1e-6, scale, out=a); step()
            eng.fc2_residual(a, wq, None, buf, scale_a=one, scale_b=scale, out=out); step()
            _, s = eng.amax_scale(out); step()
            eng.quantize_e4m3(out, s, out=a); step()
            eng.fc1_gelu(a, w1, None, scale_a=s, scale_b=scale, out_scale=one, out=hidden); step()
            eng.patchify_quantize(pixels, 16, one, out=patches); step()
            eng.fc2_residual(hidden, w2, None, out, scale_a=one, scale_b=scale, out=buf); step()

    return run, (x, y, a, hidden, patches), x0


@pytest.mark.parametrize("rows,d,ff", [(100, 256, 512), (729, 1152, 4304), (5003, 768, 3072)])
def test_back_to_back_and_captured_calls_match_synchronised_ones(engine, rows, d, ff):
    run, state, x0 = _chain(engine, rows, d, ff, seed=rows)
    run(torch.cuda.synchronize)
    want = [t.clone() for t in state]
    same = lambda: all(torch.equal(t.contiguous().view(torch.uint8), w.contiguous().view(torch.uint8)) for t, w in zip(state, want))
    for _ in range(5):
        state[0].copy_(x0)
        run(lambda: None)
        assert same()
    stream = torch.cuda.Stream()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=stream):
        state[0].copy_(x0)
        run(lambda: None)
    for _ in range(5):
        graph.replay()
        torch.cuda.synchronize()
        assert same()


def test_calls_behind_a_fork_and_a_fill_are_captured_in_order(engine):
    """What a captured launch waits for may be several nodes, and not kernels only: a fill on its own stream, work joined from another."""
    rows, d = 300, 256
    g = torch.Generator(device=DEV).manual_seed(3)
    x = torch.randn((rows, d), generator=g, device=DEV).to(torch.bfloat16)
    w = synth.quantize_e4m3(torch.randn((d, d), generator=g, device=DEV) * 0.05)[0]
    scale = torch.full((1,), 0.02, device=DEV)
    a = torch.zeros((rows, d), dtype=torch.uint8, device=DEV)
    res, out = torch.empty_like(x), torch.empty_like(x)
    want = engine.fc2_residual(engine.layernorm_quantize(x, None, None, 1e-6, scale, out=torch.zeros_like(a)), w, None, x * 2, scale_a=scale)
    main, side = torch.cuda.Stream(), torch.cuda.Stream()
    graph = torch.cuda.CUDAGraph()
    torch.cuda.synchronize()
    with torch.cuda.graph(graph, stream=main):
        a.zero_()
        engine.layernorm_quantize(x, None, None, 1e-6, scale, out=a)
        side.wait_stream(main)
        with torch.cuda.stream(side):
            res.copy_(x)
            res.mul_(2)
        main.wait_stream(side)
        engine.fc2_residual(a, w, None, res, scale_a=scale, out=out)
    for _ in range(5):
        a.fill_(0x7E)
        res.zero_()
        graph.replay()
        torch.cuda.synchronize()
        assert torch.equal(out, want)


@pytest.mark.parametrize("rows,n,k", [(100, 512, 256), (729, 1152, 4304), (3000, 4304, 1152)])
def test_weights_written_by_the_kernel_ahead(engine, rows, n, k):
    """A GEMM asks its first tile's weights into L2 before the kernel ahead has finished.  Where that kernel writes them, the GEMM
    still reads what it wrote: two weights in turn through one operand buffer, back to back and captured."""
    g = torch.Generator(device=DEV).manual_seed(rows)
    a = synth.quantize_e4m3(torch.randn((rows, k), generator=g, device=DEV))[0]
    weights = [torch.randn((n, k), generator=g, device=DEV).to(torch.bfloat16) for _ in range(2)]
    scale, res = torch.full((1,), 0.02, device=DEV), torch.randn((rows, n), generator=g, device=DEV).to(torch.bfloat16)
    b = torch.zeros((n, synth.pitch128(k)), dtype=torch.uint8, device=DEV)[:, :k]
    outs = [torch.empty((rows, n), dtype=torch.bfloat16, device=DEV) for _ in range(8)]

    def run(step):
        for i, out in enumerate(outs):
            engine.quantize_e4m3(weights[i % 2], scale, out=b); step()
            if i % 4 < 2:
                engine.fc2_residual(a, b, None, res, scale_b=scale, out=out); step()
            else:
                engine.fc1_gelu(a, b, None, scale_b=scale, out=out); step()

    run(torch.cuda.synchronize)
    want = [out.clone() for out in outs]
    assert not torch.equal(want[0], want[1]) and not torch.equal(want[2], want[3])
    stream, graph = torch.cuda.Stream(), torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=stream):
        run(lambda: None)
    for go in [lambda: run(lambda: None)] * 5 + [graph.replay] * 5:
        for out in outs:
            out.zero_()
        go()
        torch.cuda.synchronize()
        assert all(torch.equal(out, w) for out, w in zip(outs, want))
    engine.device_status()


def test_two_threads_on_their_own_streams(engine):
    """Chains of overlapped launches from two threads at once, through one handle: each stream keeps its own order."""
    chains = [_chain(engine, rows, d, ff, seed=rows) for rows, d, ff in ((729, 1152, 4304), (1300, 768, 3072))]
    wants = []
    for run, state, _ in chains:
        run(torch.cuda.synchronize)
        wants.append([t.clone() for t in state])
    errors = []

    def work(i):
        run, state, x0 = chains[i]
        stream = torch.cuda.Stream()
        try:
            with torch.cuda.stream(stream):
                for _ in range(10):
                    state[0].copy_(x0)
                    run(lambda: None)
                    stream.synchronize()
                    for t, want in zip(state, wants[i]):
                        assert torch.equal(t.contiguous().view(torch.uint8), want.contiguous().view(torch.uint8))
        except BaseException as e:      # noqa: BLE001 - handed to the test's own thread
            errors.append(e)

    torch.cuda.synchronize()
    threads = [threading.Thread(target=work, args=(i,)) for i in range(2)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    engine.device_status()
    if errors:
        raise errors[0]
