"""Convolutions whose work items outnumber the CTAs that share them: every image of a
large batch comes out as it does alone (few items, one per CTA), bit for bit. Each
output's products are added in the same order whatever the split."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("cin,cout", [(16, 16), (16, 32), (32, 16), (32, 32)])
@pytest.mark.parametrize("batch,h,w", [(40, 50, 384), (97, 7, 512), (330, 1, 128)])
def test_batch_equals_single_images(port, pg, cin, cout, batch, h, w):
    rng = np.random.default_rng(cin + 2 * cout + h)
    bf = lambda *shape: port.bf16(rng.normal(size=shape).astype(np.float32))
    x, g, mask = bf(batch, h, w, cin), bf(batch, h, w, cout), bf(batch, h, w, cin)
    wt = (rng.normal(size=(9, cout, cin)) / np.sqrt(9 * cin)).astype(np.float32)
    bias = rng.normal(size=cout).astype(np.float32)
    picks = [0, 1, batch // 2, batch - 1]
    for op, src, kw in ((pg.NN_FWD_RELU, x, {}), (pg.NN_FWD_OUT, x, {}), (pg.NN_DGRAD, g, {"aux": mask})):
        args = (wt,) if op == pg.NN_DGRAD else (wt, bias)
        whole = pg.nn_conv3x3(op, src, *args, cin=cin, cout=cout, **kw)
        assert np.any(whole != 0)
        for i in picks:
            one = {k: v[i : i + 1] for k, v in kw.items()}
            alone = pg.nn_conv3x3(op, src[i : i + 1], *args, cin=cin, cout=cout, **one)
            assert np.array_equal(whole[i], alone[0]), (op, i)
