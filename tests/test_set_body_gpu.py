"""GPU tests of set_body with another size or shape: the session or hierarchy
then steps as one that was created with that body, to the bit, in every cell
that the body touches (a dense domain's, or a hierarchy's unrefined L0 cells).
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SPHERE = dict(shape="sphere", centre=(14.3, 11.8, 12.1), a=4.0)
BOX = dict(shape="roundbox", centre=(14.3, 11.8, 12.1), a=4.0, b=3.0, c=3.5, r=1.0)
SPHEROID = dict(shape="spheroid", centre=(14.3, 11.8, 12.1), a=4.5, c=2.5)
# grown by more than a link, shrunk by more than one, and changes of shape
CHANGES = [(dict(SPHERE, a=3.0), dict(SPHERE, a=6.5)), (dict(SPHERE, a=6.5), dict(SPHERE, a=3.0)),
           (BOX, dict(SPHERE, a=5.0)), (SPHERE, BOX), (SPHEROID, dict(SPHERE, a=2.5))]


def seed(n, planar=False):
    rng = np.random.RandomState(5)
    mac = np.empty((n, 4), np.float32)
    mac[:, 0] = 1 + 0.01 * (rng.rand(n) - 0.5)
    mac[:, 1:] = 0.05 * (rng.rand(n, 3) - 0.3)
    if planar:
        mac[:, 3] = 0
    return mac


def same(x, y):
    for a, b in zip(x, y):
        assert np.array_equal(a, b)


@pytest.mark.parametrize("q", [19, 27])
@pytest.mark.parametrize("before,after", CHANGES)
def test_amr3d_l0_links_follow_the_body(lbm, q, before, after):
    dims = (40, 24, 24)
    want = np.zeros((6, 6, 10), np.uint8)
    want[1:5, 1:5, 8] = 1  # refined far from the body, which lies in L0 cells
    out = []
    for first, then in ((before, after), (after, None)):
        kw = dict(tau=0.62, has_body=1, use_bounceback=1, sponge_w=4.0, sponge_u=(0.04, 0.0, 0.0), body=first)
        a = lbm.Amr3D(lbm.amr3d_config(q, dims, refine="list", rb=4, **kw), block_want=want.ravel())
        a.init_macro(seed(int(np.prod(dims))))
        if then is not None:
            a.set_body(lbm.make_body(**then))
        a.step(4)
        out.append(a.read_coarse() + a.read_pool() + (a.forces(),))
        a.close()
    same(*out)


CIRCLE = dict(shape="ellipse", centre=(30.3, 31.8, 0.0), a=6.0, b=6.0)


@pytest.mark.parametrize("fused", [True, False])
@pytest.mark.parametrize("before,after", [(dict(CIRCLE, a=4.0, b=4.0), dict(CIRCLE, a=9.0, b=9.0)),
                                          (dict(CIRCLE, a=9.0, b=9.0), dict(CIRCLE, a=4.0, b=4.0)),
                                          (dict(CIRCLE, b=3.0, theta=0.4), CIRCLE),
                                          (CIRCLE, dict(CIRCLE, a=8.0, b=3.0))])
def test_amr2d_root_links_follow_the_body(lbm, fused, before, after):
    W, H = 128, 64
    ex = np.array([0, 1, 0, -1, 0, 1, -1, -1, 1])
    ey = np.array([0, 0, 1, 0, -1, 1, 1, -1, -1])
    w = np.array([4 / 9] + [1 / 9] * 4 + [1 / 36] * 4)
    f = np.stack([np.full(W * H, w[i] * (1 + 0.24 * ex[i] + 0.03 * ey[i]), np.float32) for i in range(9)])
    f *= (1 + 0.01 * np.random.RandomState(3).rand(9, W * H)).astype(np.float32)
    vel = np.tile(np.array([0.08, 0.01], np.float32), (W * H, 1))
    out = []
    for first, then in ((before, after), (after, None)):
        a = lbm.Amr2D(lbm.amr2d_config(W, H, tau=0.58, use_bounceback=1, sponge_w=4.0, sponge_u=(0.08, 0.0),
                                       auto_refine=0, body=first))
        a.set_fused(fused)
        a.write_root(f, vel)
        if then is not None:
            a.set_body(lbm.make_body(**then))
        a.step(5)
        a.sync()
        out.append(a.read_root())
        a.close()
    same(*out)


@pytest.mark.parametrize("before,after", CHANGES)
def test_session_links_follow_the_body(lbm, before, after):
    dims = (40, 24, 24)
    out = []
    for first, then in ((before, after), (after, None)):
        s = lbm.Solver(lbm.config_from(19, dims, tau=0.62, has_body=1, use_bounceback=1, sponge_w=4.0, body=first))
        s.init_macro(seed(int(np.prod(dims))))
        if then is not None:
            s.set_body(lbm.make_body(**then))
        s.step(4)
        out.append((s.read_f(), s.read_mac(), s.forces()))
        s.close()
    same(*out)
