"""Batches of changing view sizes on one context: a replayed graph covers the pixels of this call's views, not of the
ones it was captured with."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _views(mm, sizes, turn):
    return [(w, h, mm.scene.uniforms(w, h, yaw=turn + 23.0 * i, pitch=10.0 + i % 9, time=0.3)) for i, (w, h) in enumerate(sizes)]


@pytest.mark.parametrize("sched", ["BATCH_BLOCKS", "BATCH_PERSISTENT", "BATCH_GRAPH"])
@pytest.mark.parametrize("n", [1, 3, 75])  # 75 views: two launches of the block schedule
def test_view_sizes_change_between_calls(cuda, mmlib, sched, n):
    import marshmallow as mm
    import marshmallow.lib as L
    tex, kept = mm.render.Textures(seed=0), mm.render.Renderer()
    try:
        sizes = [[(16, 8)] * n, [(16, 8)] * (n - 1) + [(150, 70)], [(33, 17)] * n, [(20, 9)] * n,
                 [(9, 20)] * (n - 1) + [(70, 150)]]
        for k, s in enumerate(sizes):
            views = _views(mm, s, 40.0 * k)
            got = []
            for r in (kept, mm.render.Renderer()):  # the same schedule on a context of its own
                outs = [(cuda.full((h, w, 4), -7.0, device="cuda"), cuda.full((h, w), -7.0, device="cuda"))
                        for w, h, _ in views]
                r.march_batch(views, tex, outs, schedule=getattr(L, sched))
                cuda.cuda.synchronize()
                got.append([(c.cpu().numpy(), d.cpu().numpy()) for c, d in outs])
                if r is not kept:
                    r.close()
            for (c, d), (cw, dw) in zip(*got):
                assert not (cw == -7.0).any()
                assert np.array_equal(c, cw) and np.array_equal(d, dw), (k, c.shape)
    finally:
        kept.close()
        tex.close()
