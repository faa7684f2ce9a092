"""Host entry points: results that the kernel writes to the pinned buffer itself (up to 8 KB) and results that are copied, around the limit; and the
readout inside the fused kernel with one, a few and more than four graphs per CTA and round."""
import numpy as np
import pytest

from conftest import assert_close
from graphnn_b200 import engine, synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("graphs", [1, 672, 673, 1400])
def test_results(oracle_lib, graphs):
    b = synth.molecules_16k(seed=graphs, num_graphs=graphs)
    o = oracle_lib.forward(b, "oracle")
    scale = max(1.0, float(np.abs(o["logits"]).max()))
    eng = engine.S2VInference(b.weights, b.levels, device=0)
    hb = engine.build_host_batch(b)
    off = b.graph_offsets().astype(np.int32)
    for _ in range(2):
        logits, pred = eng.infer_host(hb)
        assert_close(logits, o["logits"], "csr", scale)
        assert np.array_equal(pred, logits.argmax(1))
        logits, pred = np.full_like(o["logits"], np.nan), np.full(graphs, -1, np.int32)
        eng.ctx.infer_edges_host(eng.model, graphs, b.num_nodes, b.edge_src.astype(np.int32), b.edge_dst.astype(np.int32), off, b.tags.astype(np.int32),
                                 logits, pred)
        assert_close(logits, o["logits"], "edges", scale)
        assert np.array_equal(pred, logits.argmax(1))


@pytest.mark.parametrize("graphs", [64, 700, 1500])
def test_readout_inside(oracle_lib, graphs):
    """Small graphs at d = 64, several graphs per CTA, through the one launch."""
    b = synth.mutag_like(seed=graphs, num_graphs=graphs)
    o = oracle_lib.forward(b, "oracle")
    eng = engine.S2VInference(b.weights, b.levels, device=0)
    db = eng.to_device(engine.build_host_batch(b))
    n0 = eng.ctx.launches
    logits, probs, pred, _ = eng.forward(db)
    eng.ctx.synchronize()
    assert eng.ctx.launches - n0 == 1
    assert_close(logits.cpu().numpy(), o["logits"], "logits", max(1.0, float(np.abs(o["logits"]).max())))
    assert_close(probs.cpu().numpy().sum(1), np.ones(graphs), "probabilities")
