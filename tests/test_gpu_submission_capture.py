"""A program that captures a graph of its own may go on submitting meanwhile: submissions with resident bindings ask nothing that a capture in
progress forbids its process."""
import numpy as np
import pytest

import vyre_b200 as vb

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


def test_chained_submissions_during_a_capture():
    d, m, k = vb.Device.acquire(0), 256, 1024
    prog = vb.linear_rows_no_bias("x", "w", "out", m, k, k)
    sess = vb.ArtifactSession.compile(prog, d)
    slots = {b["name"]: b["binding"] for b in prog.buffers()}
    rng = np.random.default_rng(3)
    x, w = (d.resident_from(rng.standard_normal(n).astype(np.float32)) for n in (m * k, k * k))
    outs, chain = [d.allocate_resident(4 * m * k) for _ in range(6)], []
    for o in outs:
        bs = vb.BindingSet(sess.artifact.digest())
        for name, h in (("x", x), ("w", w), ("out", o)):
            bs.insert_resident(slots[name], h)
        chain.append(bs)
    for _ in range(2):  # what a first submission allocates is there
        for sub in [sess.submit(bs, leave_resident=True) for bs in chain]:
            assert sub.wait().device_ns > 0
    want = d.download_resident(outs[0], 4 * m * k).tobytes()
    t, g = torch.zeros(8, device="cuda"), torch.cuda.CUDAGraph()
    torch.cuda.synchronize()
    with torch.cuda.graph(g):
        t.add_(1)
        subs = [sess.submit(bs, leave_resident=True) for bs in chain]  # all but the first find one pending
        t.add_(1)
    done = [s.wait() for s in subs]
    assert all(0 < c.device_ns < 50_000_000 for c in done)
    assert all(d.download_resident(o, 4 * m * k).tobytes() == want for o in outs)
    g.replay()
    torch.cuda.synchronize()
    assert (t == 2).all()
    del done, subs, sess
    for h in [x, w] + outs:
        d.free_resident(h)
    d.release()
