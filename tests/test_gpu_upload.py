"""Uploads from page-locked and pageable host arrays, with and without masses:
the same device layout, charges and masses either way."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("masses", [None, "ones", "last", "mixed"])  # "last": only the last particle's differs from 1
@pytest.mark.parametrize("n", [1, 255, 257, 70001])
def test_pageable_equals_page_locked(pg, n, masses):
    rng = np.random.default_rng(n)
    a = {"x": rng.random(n) * 20, "y": rng.random(n) * 12, "vx": rng.normal(size=n), "vy": rng.normal(size=n),
         "q": rng.choice([-1.0, 0.5], n)}
    if masses:
        a["m"] = np.ones(n)
        if masses == "last":
            a["m"][-1] = 3.0
        if masses == "mixed":
            a["m"] = rng.random(n) + 0.5
    out = []
    for pinned in (False, True, "m pageable"):
        hold = {}
        args = {}
        for k, v in a.items():
            if pinned and not (k == "m" and pinned == "m pageable"):
                hold[k] = pg.PinnedArray(n)
                hold[k].array[:] = v
                args[k] = hold[k].array
            else:
                args[k] = v
        with pg.Context(20, 12, 20.0, 12.0, n) as c:
            c.upload(**args)
            out.append((c.device_layout(), c.download()))
        args.clear()
        for h in hold.values():
            h.free()
    for lay, host in out[1:]:
        for k in lay:
            assert np.array_equal(lay[k], out[0][0][k])
        for k in host:
            assert np.array_equal(host[k], out[0][1][k])
    want = a.get("m", np.ones(n)).astype(np.float32)
    assert np.array_equal(out[0][1]["m"], want)


def test_mass_set_then_cleared(pg):
    """A set with masses, then one without: the gather divides by the new set's masses."""
    n = 1000
    rng = np.random.default_rng(5)
    x, y, v = rng.random(n) * 16, rng.random(n) * 16, rng.normal(size=n)
    e = rng.normal(size=256)
    got = []
    for first in (None, rng.random(n) + 0.5):
        with pg.Context(16, 16, 16.0, 16.0, n) as c:
            if first is not None:
                c.upload(x, y, -np.ones(n), v, v, first)
            c.upload(x, y, -np.ones(n), v, v, np.ones(n))
            c.set_fields(ex=e, ey=e)
            c.gather(0.1)
            got.append(c.device_layout()["vx"])
            assert np.all(c.download()["m"] == 1.0)
    assert np.array_equal(*got)


@pytest.mark.parametrize("shift", [1, 4, 8])
def test_upload_from_any_byte_address(pg, shift):
    """Arrays whose elements do not lie on multiples of their size are copied first."""
    n = 777
    rng = np.random.default_rng(shift)
    a = {"x": rng.random(n) * 16, "y": rng.random(n) * 8, "q": rng.choice([-1.0, 0.5], n), "m": rng.random(n) + 0.5}
    out = []
    for s in (0, shift):
        args = {}
        for k, v in a.items():
            raw = np.zeros(n * 8 + 16, np.uint8)
            off = (-raw.ctypes.data) % 16 + s
            raw[off : off + n * 8] = np.frombuffer(v.tobytes(), np.uint8)
            args[k] = raw[off : off + n * 8].view(np.float64)
        with pg.Context(16, 8, 16.0, 8.0, n) as c:
            c.upload(**args)
            out.append((c.device_layout(), c.download()))
    for i in (0, 1):
        for k in out[0][i]:
            assert np.array_equal(out[0][i][k], out[1][i][k])


def test_network_gradient_from_any_host_array(pg):
    """Loss and gradient of fields that the kernels read in place (pageable, page-locked)
    and of fields that are copied first (not on a multiple of 4 bytes): the same bits."""
    nx, ny, batch = 128, 8, 3
    n = batch * nx * ny
    rng = np.random.default_rng(2)
    fields = [rng.normal(size=(batch, ny, nx)).astype(np.float32) for _ in range(2)]
    hold = [pg.PinnedArray(n // 2) for _ in range(2)]
    odd = []
    for h, f in zip(hold, fields):
        h.array.view(np.float32)[:] = f.reshape(-1)
        raw = np.zeros(4 * n + 16, np.uint8)
        off = (-raw.ctypes.data) % 16 + 1
        raw[off : off + 4 * n] = np.frombuffer(f.tobytes(), np.uint8)
        odd.append(raw[off : off + 4 * n].view(np.float32).reshape(f.shape))
    pinned = [h.array.view(np.float32).reshape(batch, ny, nx) for h in hold]
    with pg.Context(nx, ny, float(nx), float(ny), 16) as c:
        c.ws_init(seed=3)
        got = [c.ws_loss_grad(*a) for a in (fields, odd, pinned, (fields[0], odd[1]), (pinned[0], fields[1]))]
    del pinned
    for h in hold:
        h.free()
    for loss, grad in got[1:]:
        assert loss == got[0][0]
        assert np.array_equal(grad, got[0][1])
