"""Batches whose edges join two graphs.  The host entry points know the largest graph and so would keep whole graphs in shared memory,
but nobody promised them separate graphs: the results are those of the matrix as given, wherever the two graphs end up."""
import numpy as np
import pytest
import torch

from conftest import assert_close
from graphnn_b200 import engine
from test_graph_fused_gpu import f64, make

pytestmark = pytest.mark.gpu


def crossing(sizes, d, joins, seed):
    b = make(sizes, 2.2, d, 9, 3, 64, 3, seed=seed)
    off = b.graph_offsets()
    extra = [(off[g] + i, off[h] + j) for g, i, h, j in joins]
    b.edge_src = np.concatenate([b.edge_src, [u for u, v in extra]]).astype(np.int32)
    b.edge_dst = np.concatenate([b.edge_dst, [v for u, v in extra]]).astype(np.int32)
    return b


def check(b, logits, pred):
    rp, ci = engine.capi.build_n2n_csr_host(b.num_nodes, b.edge_src, b.edge_dst, with_val=False)[:2]
    _, want = f64(b, rp, ci, None, None, False)
    assert_close(logits, want, "logits", scale=max(1.0, float(np.abs(want).max())))
    assert np.array_equal(pred, logits.argmax(1))


@pytest.mark.parametrize("validate", [0, 1])
@pytest.mark.parametrize("d", [32, 64, 128])
@pytest.mark.parametrize("sizes,joins", [
    ([30, 40, 20], [(0, 1, 1, 2)]),                                  # neighbours that may share a tile
    ([30] * 900, [(0, 0, 899, 29), (450, 3, 451, 4)]),               # far apart
    ([100] * 20, [(3, 0, 4, 0), (4, 0, 3, 0)]),
])
def test_host_entry_points(sizes, joins, d, validate):
    b = crossing(sizes, d, joins, seed=d)
    eng = engine.S2VInference(b.weights, b.levels)
    eng.ctx.set_option(eng.ctx.OPT_VALIDATE_HOST_INPUT, validate)
    hb = engine.build_host_batch(b)
    assert hb.max_graph_nodes == 0
    plain = make(sizes, 2.2, d, 9, 3, 64, 3, seed=d)                  # the same without the joins: the context carries nothing over
    for batch in (b, plain, b):
        check(batch, *eng.infer_host(engine.build_host_batch(batch)))
        logits, pred = np.empty((b.num_graphs, 3), np.float32), np.empty(b.num_graphs, np.int32)
        eng.ctx.infer_edges_host(eng.model, b.num_graphs, b.num_nodes, np.ascontiguousarray(batch.edge_src, np.int32),
                                 np.ascontiguousarray(batch.edge_dst, np.int32), hb.graph_ptr.numpy(), hb.tags.numpy(), logits, pred)
        check(batch, logits, pred)
    logits, _, pred, _ = eng.forward(eng.to_device(hb))
    eng.ctx.synchronize()
    check(b, logits.cpu().numpy(), pred.cpu().numpy())


@pytest.mark.parametrize("which", [(1, 0), (0, 1), (1, 1)])
def test_two_lanes(which):
    batches = [crossing([90] * 60, 64, [(0, 0, 59, 5)] if w else [], seed=3 + i) for i, w in enumerate(which)]
    eng = engine.S2VInference(batches[0].weights, batches[0].levels)
    jobs = []
    for b in batches:
        b.weights = batches[0].weights
        hb = engine.build_host_batch(b)
        pin = lambda a: torch.from_numpy(np.ascontiguousarray(a, np.int32)).pin_memory()
        jobs.append((pin(b.edge_src), pin(b.edge_dst), hb.graph_ptr.pin_memory(), hb.tags.pin_memory(),
                     np.empty((60, 3), np.float32), np.empty(60, np.int32)))
    for _ in range(3):
        for lane, (b, (es, ed, gp, tg, logits, pred)) in enumerate(zip(batches, jobs)):
            logits[:] = np.nan
            eng.ctx.infer_edges_host_submit(lane, eng.model, 60, b.num_nodes, es.numpy(), ed.numpy(), gp.numpy(), tg.numpy(), logits, pred)
        for lane, (b, j) in enumerate(zip(batches, jobs)):
            eng.ctx.infer_host_wait(lane)
            check(b, j[4], j[5])
