"""Host entry points: every call hands over its own batch's results, on both sides of the size up to which the kernel writes them to the pinned
buffer (8 KB, 672 graphs of two classes).  Batches of one size with other graphs take turns, so that what an earlier call left there would show."""
import numpy as np
import pytest
import torch

from conftest import assert_close
from graphnn_b200 import engine, synth

pytestmark = pytest.mark.gpu
i32 = lambda a: np.ascontiguousarray(a, np.int32)


def pair(oracle_lib, graphs):
    batches = [synth.molecules_16k(seed=s, num_graphs=graphs) for s in (2, 3)]
    batches[1].weights = batches[0].weights
    want = [oracle_lib.forward(b, "oracle")["logits"] for b in batches]
    assert not np.allclose(want[0], want[1], rtol=1e-3)
    return batches, want


def check(logits, pred, want, what):
    if logits is not None:
        assert_close(logits, want, what, max(1.0, float(np.abs(want).max())))
    if pred is not None:
        best = np.sort(want, 1)
        clear = best[:, -1] - best[:, -2] > 1e-3 * max(1.0, float(np.abs(want).max()))   # (two classes this close may be taken either way)
        assert np.array_equal(pred[clear], want.argmax(1)[clear]), what


@pytest.mark.parametrize("graphs", [3, 672, 673])
@pytest.mark.parametrize("logits,pred", [(True, True), (True, False), (False, True)])
def test_taking_turns(oracle_lib, graphs, logits, pred):
    batches, want = pair(oracle_lib, graphs)
    eng = engine.S2VInference(batches[0].weights, batches[0].levels)
    hosts = [engine.build_host_batch(b) for b in batches]
    for turn in range(4):
        b, w, hb = batches[turn % 2], want[turn % 2], hosts[turn % 2]
        for entry in ("csr", "edges"):
            out = np.full((graphs, 2), np.nan, np.float32) if logits else None
            best = np.full(graphs, -1, np.int32) if pred else None
            if entry == "csr":
                cb = eng.ctx.make_batch(graphs, hb.num_nodes, hb.row_ptr, hb.col_idx, None, hb.graph_ptr, hb.tags, None)
                eng.ctx.infer_host(eng.model, cb, out, best)
            else:
                eng.ctx.infer_edges_host(eng.model, graphs, b.num_nodes, i32(b.edge_src), i32(b.edge_dst), i32(b.graph_offsets()), i32(b.tags), out, best)
            check(out, best, w, f"{entry}, turn {turn}")
            b, w, hb = batches[1 - turn % 2], want[1 - turn % 2], hosts[1 - turn % 2]   # (the other entry point shares the buffer)


@pytest.mark.parametrize("graphs", [672, 673])
def test_two_lanes_taking_turns(oracle_lib, graphs):
    batches, want = pair(oracle_lib, graphs)
    eng = engine.S2VInference(batches[0].weights, batches[0].levels)
    pin = lambda a: torch.from_numpy(i32(a)).pin_memory().numpy()
    jobs = [tuple(pin(a) for a in (b.edge_src, b.edge_dst, b.graph_offsets(), b.tags)) for b in batches]
    for turn in range(4):
        outs = []
        for lane in (0, 1):
            k = (turn + lane) % 2
            outs.append((np.full((graphs, 2), np.nan, np.float32), np.full(graphs, -1, np.int32), k))
            eng.ctx.infer_edges_host_submit(lane, eng.model, graphs, batches[k].num_nodes, *jobs[k], *outs[lane][:2])
        for lane in (0, 1):
            eng.ctx.infer_host_wait(lane)
            check(*outs[lane][:2], want[outs[lane][2]], f"lane {lane}, turn {turn}")
