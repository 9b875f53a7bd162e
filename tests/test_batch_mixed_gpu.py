"""Batches whose layers take both the shift kernel and the fused kernel: a capture
runs them as two branches, which a replay joins before what follows it."""
import pytest

import test_shift_conv as base

pytestmark = pytest.mark.gpu

# n, c, h, w, k: 925 MFLOP (the shift kernel's table), 578 MFLOP of rows too long for
# it (a launch of its own), small layers of the fused kernel
SHAPES = [(2, 64, 56, 56, 128), (1, 16, 40, 224, 224), (2, 512, 7, 7, 512), (2, 32, 15, 15, 48)]


@pytest.mark.parametrize("picks", [(0, 2, 3), (0, 1, 2), (1, 3), (0, 1)])
def test_replays_join_before_what_follows(wino, cuda, picks):
    import torch
    cases = [base._fused_case(cuda, SHAPES[i], 30 + i) for i in picks]
    b, layers = wino.Batch(), []
    for x, wt, _, res in cases:
        n, c, h, w = x.shape
        k = wt.shape[0]
        ws = torch.empty(wino.fused_conv_workspace_bytes(n, c, h, w, k), dtype=torch.uint8, device=cuda)
        y, u = torch.empty_like(res), wino.filter_transform(wt)
        b.add(x, u, k, y, workspace=ws)
        layers.append((x, u, k, y))
    torch.cuda.synchronize()
    b.capture()
    streams = [torch.cuda.Stream(), torch.cuda.Stream()]
    got = []
    for i in range(6):
        # inputs rewritten and outputs read on the replay's stream, no other wait
        s = streams[i & 1]
        s.wait_stream(streams[1 - (i & 1)])
        with torch.cuda.stream(s):
            for x, _, _, _ in layers:
                x.mul_(-0.5)
            b.launch(stream=s)
            got.append([(x.clone(), y.clone()) for x, _, _, y in layers])
            for _, _, _, y in layers:
                y.fill_(float("nan"))
    torch.cuda.synchronize()
    for pass_ in got:
        for (_, u, k, _), (x, y) in zip(layers, pass_):
            assert torch.equal(y, wino.conv2d_fused(x, u, k))
    b.close()
    assert wino.error_read_clear() == 0


def test_a_callers_graph_outlives_layers_added_later(wino, cuda):
    """A run captured into the caller's own graph replays after the batch grew: the
    operands of the layers it holds stay where they are."""
    import torch
    shapes = [(2, 64, 56, 56, 128), (8, 128, 28, 28, 128), (8, 256, 14, 14, 256)]
    cases = [base._fused_case(cuda, s, 40 + i) for i, s in enumerate(shapes)]
    b, layers = wino.Batch(), []

    def add(case):
        x, wt, _, res = case
        n, c, h, w = x.shape
        ws = torch.empty(wino.fused_conv_workspace_bytes(n, c, h, w, wt.shape[0]), dtype=torch.uint8, device=cuda)
        layers.append((x, wino.filter_transform(wt), wt.shape[0], torch.empty_like(res), ws))
        b.add(layers[-1][0], layers[-1][1], layers[-1][2], layers[-1][3], workspace=ws)

    add(cases[0])
    b.run()
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        b.run()
    for case in cases[1:]:
        add(case)
        b.run()
    x, u, k, y, _ = layers[0]
    for _ in range(2):
        x.mul_(-0.5)
        y.fill_(float("nan"))
        graph.replay()
        torch.cuda.synchronize()
        assert torch.equal(y, wino.conv2d_fused(x, u, k))
    b.run()
    torch.cuda.synchronize()
    for x, u, k, y, _ in layers:
        assert torch.equal(y, wino.conv2d_fused(x, u, k))
    b.close()
    assert wino.error_read_clear() == 0


def test_tuner_reports_only_what_it_ran(wino, cuda):
    """The shift kernel has no configurations: one time for its layer, the others
    -1; the fused kernel's layer has one for each configuration without splits."""
    import torch
    b, keep = wino.Batch(), []
    for i, shape in enumerate([(2, 64, 56, 56, 128), (2, 64, 14, 14, 64)]):
        x, wt, _, res = base._fused_case(cuda, shape, 50 + i)
        n, c, h, w, k = shape
        ws = torch.empty(wino.fused_conv_workspace_bytes(n, c, h, w, k), dtype=torch.uint8, device=cuda)
        keep.append((x, wino.filter_transform(wt), res, ws))
        b.add(x, keep[-1][1], k, res, workspace=ws)
    rows, _ = b.tune(reps=1)
    ran = [[c for c, t in enumerate(row) if t > 0] for row in rows]
    assert len(ran[0]) == 1 and ran[0][0] == b.config(0)
    assert len(ran[1]) > 1 and b.config(1) in ran[1]
    assert all(t == -1 for row, r in zip(rows, ran) for c, t in enumerate(row) if c not in r)
    b.close()
    assert wino.error_read_clear() == 0
