"""Several host threads, each with a context and a stream of its own, at sizes that need different amounts of shared memory from the
same kernels: every call succeeds and gives the results of the same calls one after the other."""
import threading

import pytest
import torch

from graphnn_b200 import engine
from test_graph_fused_gpu import make

pytestmark = pytest.mark.gpu


def test_contexts_of_several_threads():
    jobs = []
    for i in range(8):
        # one kernel, tiles of 256 and of 640 rows; dense inputs: 5 and 25 attributes
        b = make([200, 3] if i % 2 else [600, 7], 2.2, 64, 25 if i % 4 < 2 else 5, 2, 20 + 12 * (i % 3), 2, seed=i)
        eng = engine.S2VInference(b.weights, b.levels)
        db = eng.to_device(engine.build_host_batch(b), b.dense_x())
        torch.cuda.synchronize()
        logits, _, _, _ = eng.forward(db)
        eng.ctx.synchronize()
        want = logits.clone()
        args = (torch.empty_like(logits), torch.empty_like(logits), torch.empty(b.num_graphs, dtype=torch.int32, device="cuda"))
        cb = eng.ctx.make_batch(db.num_graphs, db.num_nodes, db.row_ptr, db.col_idx, None, db.graph_ptr, None, db.x_dense, db.max_graph_nodes)
        jobs.append((eng, db, cb, eng._workspace(db.num_nodes, db.num_graphs), want, args))
    torch.cuda.synchronize()
    errors = []
    start = threading.Barrier(len(jobs))

    def work(i):
        eng, _, cb, ws, want, (logits, probs, pred) = jobs[i]
        try:
            start.wait()
            for _ in range(2000):
                eng.ctx.forward(eng.model, cb, ws, logits, probs, pred, None)
            eng.ctx.synchronize()
            if not torch.equal(logits, want):
                errors.append(f"thread {i}: other results")
        except Exception as e:                              # noqa: BLE001 (reported by the test's own thread)
            errors.append(f"thread {i}: {e}")

    threads = [threading.Thread(target=work, args=(i,)) for i in range(len(jobs))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors
