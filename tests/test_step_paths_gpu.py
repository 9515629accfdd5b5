"""GPU tests of the step's alternative paths: whichever path a size, storage
or topology selects, a cell gets the same bits.

* 3D dense launch mappings (rows, or a plane's cells as one run) and block
  kinds, against the same domain in a batch, which updates one cell per
  thread by plain indices;
* the D2Q9 reach box, against the batch, which evaluates the body everywhere;
* a moving window whose rows are no whole number of launch blocks, the body on
  either side of the seam, against the oracle;
* a free body that is pinned, against the prescribed pose;
* 3D AMR macro-steps over the live chunks only, against single macro-steps,
  whose last substep covers every tile cell;
* the fused 2D AMR macro-steps with more tiles than blocks, against the six
  launches.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def dense_and_batch(lbm, q, dims, steps, seed=0, **kw):
    n = int(np.prod(dims))
    rng = np.random.RandomState(seed)
    mac = np.empty((n, 4), np.float32)
    mac[:, 0] = 1 + 0.01 * (rng.rand(n) - 0.5)
    mac[:, 1:] = 0.05 * (rng.rand(n, 3) - 0.3)
    if q == 9:
        mac[:, 3] = 0
    cfg = lbm.config_from(q, dims, **kw)
    s, b = lbm.Solver(cfg), lbm.Batch([cfg])
    s.init_macro(mac)
    b.init_macro(0, mac)
    s.step(steps)
    b.step(steps)
    assert np.array_equal(s.read_f(), b.read_f(0))
    assert np.array_equal(s.read_mac(), b.read_mac(0))
    f, g = s.forces(), b.forces()[0]
    # FP64 sums of the same cell contributions, differently grouped
    assert np.allclose(f, g, rtol=1e-10, atol=1e-12 * max(np.abs(g).max(), 1e-300))
    s.close()
    b.close()
    return f


BODY = dict(has_body=1, use_bounceback=1, sponge_w=4.0, sponge_u=(0.04, 0.0, 0.0), force=(1e-6, 0.0, 0.0))
# edges of the 64- and 128-cell blocks, odd rows (no word holds two cells),
# the smallest rows, planes of an odd number of cells
DIMS = [(3, 3, 3), (4, 3, 5), (5, 5, 3), (63, 7, 5), (64, 6, 5), (65, 5, 7), (100, 9, 6), (127, 5, 5), (128, 4, 6),
        (129, 5, 3), (130, 6, 4), (151, 7, 5), (256, 3, 4)]


@pytest.mark.parametrize("storage", ["fp32", "fp16", "bf16"])
@pytest.mark.parametrize("dims", DIMS)
def test_fluid_domain_equals_batch(lbm, dims, storage):
    dense_and_batch(lbm, 19, dims, 4, tau=0.6, force=(1e-5, -2e-5, 3e-6), storage=storage)


@pytest.mark.parametrize("storage", ["fp32", "fp16", "bf16"])
@pytest.mark.parametrize("q,trt,dims", [(19, 0, (66, 24, 22)), (19, 1, (51, 23, 20)), (27, 0, (100, 26, 24)),
                                        (27, 1, (128, 20, 25)), (27, 1, (37, 30, 21))])
def test_body_domain_equals_batch(lbm, q, trt, dims, storage):
    body = dict(shape="sphere", centre=(dims[0] / 3.0, dims[1] / 2.0, dims[2] / 2.0), a=4.0)
    f = dense_and_batch(lbm, q, dims, 5, tau=0.58, storage=storage, trt=trt, trt_lambda=0.1875, body=body, **BODY)
    assert abs(f[0]) > 0


@pytest.mark.parametrize("storage", ["fp32", "bf16"])
@pytest.mark.parametrize("q,trt,dims,shape", [(19, 0, (66, 24, 22), "sphere"), (27, 0, (64, 26, 24), "roundbox"),
                                              (19, 1, (100, 21, 20), "spheroid"), (27, 1, (3, 4, 5), "sphere")])
def test_penalty_domain_equals_batch(lbm, q, trt, dims, shape, storage):
    body = dict(shape=shape, centre=(dims[0] / 3.0, dims[1] / 2.0, dims[2] / 2.0), a=4.0, b=3.0, c=3.0,
                r=1.0 if shape == "roundbox" else 0.0, quat=(0.96, 0.28, 0.0, 0.0), v=(0.01, 0.0, 0.0))
    f = dense_and_batch(lbm, q, dims, 5, tau=0.58, storage=storage, trt=trt, trt_lambda=0.1875, wall=(0, 1, 0),
                        body=body, **dict(BODY, use_bounceback=0))
    assert abs(f[0]) > 0


@pytest.mark.parametrize("storage", ["fp32", "fp16"])
def test_walls_and_body_at_the_edge_equal_batch(lbm, storage):
    body = dict(shape="roundbox", centre=(3.0, 20.5, 2.0), a=4.0, b=3.0, c=3.0, r=1.0, quat=(0.96, 0.28, 0.0, 0.0))
    f = dense_and_batch(lbm, 19, (70, 22, 18), 5, tau=0.6, storage=storage, wall=(1, 1, 1), body=body, has_body=1,
                        use_bounceback=1)
    assert abs(f[0]) > 0


def test_spheroid_links_equal_batch_and_oracle_side(lbm):
    body = dict(shape="spheroid", centre=(15.3, 11.8, 12.1), a=5.0, c=2.5, quat=(0.9, 0.3, 0.3, 0.1))
    qn = np.linalg.norm(body["quat"])
    body["quat"] = tuple(v / qn for v in body["quat"])
    f = dense_and_batch(lbm, 19, (40, 24, 24), 6, tau=0.6, body=body, **BODY)
    assert abs(f[0]) > 0


@pytest.mark.parametrize("storage", ["fp32", "bf16"])
@pytest.mark.parametrize("bb", [0, 1])
@pytest.mark.parametrize("body", [dict(centre=(40.0, 30.0, 0.0), a=5.0, b=5.0),
                                  dict(centre=(3.0, 30.5, 0.0), a=6.0, b=3.0, theta=0.4),
                                  dict(centre=(100.2, 58.7, 0.0), a=4.0, b=4.0, v=(0.01, 0.0, 0.0), w=(0.0, 0.0, 0.01))])
def test_2d_reach_box_equals_batch(lbm, body, bb, storage):
    f = dense_and_batch(lbm, 9, (130, 61, 1), 6, tau=0.6, storage=storage, has_body=1, use_bounceback=bb,
                        sponge_w=4.0, sponge_u=(0.04, 0.0, 0.0), body=dict(shape="ellipse", **body))
    assert abs(f[0]) > 0


@pytest.mark.parametrize("nx,cx", [(100, 1.3), (100, 97.7), (130, 8.25), (130, 126.6), (70, 69.9)])
def test_windowed_force_across_a_ragged_seam(lbm, oracle, nx, cx):
    dims = (nx, 24, 22)
    rng = np.random.RandomState(2)
    mac = np.empty((int(np.prod(dims)), 4), np.float32)
    mac[:, 0] = 1 + 0.01 * (rng.rand(len(mac)) - 0.5)
    mac[:, 1:] = 0.04 * (rng.rand(len(mac), 3) - 0.5)
    f0 = oracle.init_eq(19, mac, fp32=True)
    cfg = lbm.config_from(19, dims, tau=0.6, has_body=1, use_bounceback=1, sponge_w=4.0, window="x", win_anchor=(30, 0, 0),
                          body=dict(shape="sphere", centre=(cx, 11.5, 11.0), a=6.0, v=(0.1, 0.0, 0.0)))
    s = lbm.Solver(cfg)
    s.write_f(f0.astype(np.float32))
    s.step(3)
    g = s.forces()
    s.close()
    o = oracle.run(cfg, f0, 3)[2][-1, :6]
    assert np.abs(g - o).max() <= 1e-4 * max(np.abs(o).max(), 1e-3)  # the bound of the seam test at whole blocks


@pytest.mark.parametrize("storage", ["fp32", "fp16"])
@pytest.mark.parametrize("shape,bb", [("sphere", 1), ("spheroid", 1), ("roundbox", 1), ("spheroid", 0)])
def test_pinned_free_body_equals_prescribed_pose(lbm, shape, bb, storage):
    dims = (75, 30, 28)
    n = int(np.prod(dims))
    body = dict(shape=shape, centre=(22.3, 14.6, 13.9), a=5.0, b=4.0, c=3.0, r=1.0 if shape == "roundbox" else 0.0,
                quat=(0.8, 0.6, 0.0, 0.0))
    cfg = lbm.config_from(19, dims, tau=0.6, storage=storage, body=body, **dict(BODY, use_bounceback=bb))
    out = []
    for free in (False, True):
        s = lbm.Solver(cfg)
        mac = np.tile(np.array([1.0, 0.04, 0.0, 0.0], np.float32), (n, 1))
        s.init_macro(mac)
        if free:
            s.set_free_body(lbm.body_state(cfg.body, 1.0), lbm.body_opts(pinned=1))
        s.step(6)
        out.append((s.read_f(), s.read_mac(), s.forces()))
        s.close()
    assert np.array_equal(out[0][0], out[1][0])
    assert np.array_equal(out[0][1], out[1][1])
    assert np.allclose(out[0][2], out[1][2], rtol=1e-10, atol=1e-12 * np.abs(out[0][2]).max())


@pytest.mark.parametrize("storage", ["fp32", "fp16"])
@pytest.mark.parametrize("dims", [(3, 3, 1), (4, 257, 1), (1625, 40, 1), (37838, 3, 1), (37837, 3, 1), (70001, 5, 1)])
def test_2d_rows_of_any_length_equal_batch(lbm, dims, storage):
    """The batch finds a cell's row by a multiplication, exact on its own up to
    nx^2 ny = 2^32 (between the fourth and the fifth of these domains)."""
    dense_and_batch(lbm, 9, dims, 3, tau=0.6, force=(1e-5, -2e-5, 0.0), storage=storage, wall=(0, 1, 0), sponge_w=4.0)


QUAT = (0.8, 0.36, 0.48, 0.0)


@pytest.mark.parametrize("storage", ["fp32", "fp16"])
@pytest.mark.parametrize("body", [dict(shape="sphere", a=4.0), dict(shape="sphere", a=4.0, quat=QUAT),
                                  dict(shape="spheroid", a=5.0, c=2.5, quat=QUAT),
                                  dict(shape="roundbox", a=5.0, b=3.0, c=3.5, r=1.0, quat=QUAT),
                                  dict(shape="sphere", a=12.5), dict(shape="roundbox", a=11.0, b=11.0, c=11.0, r=2.0)])
@pytest.mark.parametrize("q,trt,dims,window,cx", [(19, 0, (130, 30, 28), "x", 4.3), (27, 1, (64, 27, 40), "xyz", 61.7),
                                                  (19, 1, (96, 40, 26), "yz", 40.2)])
def test_windowed_step_equals_the_general_update(lbm, q, trt, dims, window, cx, body, storage):
    """A prescribed body's windowed step runs its fluid blocks apart and tests
    its links in the body's frame where they see one image of it (not about the
    largest bodies here, which reach half-way round an axis); a free body's,
    here pinned to the same pose, updates every cell alike, with the distance
    of each source."""
    n = int(np.prod(dims))
    rng = np.random.RandomState(4)
    mac = np.empty((n, 4), np.float32)
    mac[:, 0] = 1 + 0.01 * (rng.rand(n) - 0.5)
    mac[:, 1:] = 0.04 * (rng.rand(n, 3) - 0.4)
    body = dict(body, centre=(cx, dims[1] - 2.4, 3.7))
    cfg = lbm.config_from(q, dims, tau=0.6, storage=storage, trt=trt, trt_lambda=0.1875, window=window,
                          win_anchor=(20, 11, 12), body=body, **dict(BODY, sponge_w=6.0))
    out = []
    for free in (False, True):
        s = lbm.Solver(cfg)
        s.init_macro(mac)
        if free:
            s.set_free_body(lbm.body_state(cfg.body, 1.0), lbm.body_opts(pinned=1))
        s.step(5)
        out.append((s.read_f(), s.read_mac(), s.forces()))
        s.close()
    assert np.array_equal(out[0][0], out[1][0])
    assert np.array_equal(out[0][1], out[1][1])
    assert np.allclose(out[0][2], out[1][2], rtol=1e-10, atol=1e-12 * np.abs(out[0][2]).max())


@pytest.mark.parametrize("q,rb,dynamic,shape", [(19, 4, 0, "roundbox"), (27, 4, 0, "sphere"), (19, 2, 0, "sphere"),
                                                (19, 3, 0, "roundbox"), (19, 4, 1, "sphere")])
def test_amr3d_live_chunks_equal_whole_tiles(lbm, q, rb, dynamic, shape):
    from getting_air_b200 import scenarios as sc
    dims = (12 * rb, 8 * rb, 8 * rb)
    kw = dict(tau=0.62, has_body=1, use_bounceback=1, sponge_w=4.0, sponge_u=(0.04, 0.0, 0.0),
              body=dict(shape=shape, centre=(4.3 * rb, 4.0 * rb, 3.9 * rb), a=1.6 * rb, b=1.4 * rb, c=1.4 * rb,
                        r=0.3 * rb if shape == "roundbox" else 0.0, v=(0.2 if dynamic else 0.0, 0.0, 0.0)))
    runs = []
    for single in (False, True):
        a = lbm.Amr3D(lbm.amr3d_config(q, dims, refine="body", rb=rb, margin=2.0, dynamic=dynamic, manage_every=3,
                                       slot_headroom=2.0, **kw))
        a.init_macro(sc.uniform_macro(int(np.prod(dims)), (0.04, 0.0, 0.0)))
        for _ in range(2):
            for k in range(7 if single else 1):
                a.step(1 if single else 7)
            body = lbm.make_body(**dict(kw["body"], centre=(4.3 * rb + (3.0 if dynamic else 0.0), 4.0 * rb, 3.9 * rb)))
            a.set_body(body)
        runs.append(a.read_coarse() + a.read_pool() + (a.forces(), a.topology()["block_slot"]))
        a.close()
    for x, y in zip(*runs):
        assert np.array_equal(x, y)
    assert abs(runs[0][4][0]) > 0


@pytest.mark.parametrize("dynamic", [0, 1])
@pytest.mark.parametrize("vx", [0.0, 0.1])
def test_amr3d_work_lists_of_many_tiles(lbm, dynamic, vx):
    """As above with more tiles than one CTA builds the lists of (1024),
    a body at rest and a moving one, whose solid inside is most of the tiles.
    Calls of one macro-step right after set_body run without the lists."""
    from getting_air_b200 import scenarios as sc
    dims = (56, 40, 40)
    body = dict(shape="roundbox", centre=(20.3, 20.0, 19.9), a=11.0, b=11.0, c=11.0, r=2.0, v=(vx, 0.0, 0.0))
    runs = []
    for single in (False, True):
        a = lbm.Amr3D(lbm.amr3d_config(19, dims, refine="body", rb=2, margin=2.0, dynamic=dynamic, manage_every=2,
                                       slot_headroom=1.5, tau=0.62, has_body=1, use_bounceback=1, sponge_w=4.0,
                                       sponge_u=(0.04, 0.0, 0.0), body=body))
        a.init_macro(sc.uniform_macro(int(np.prod(dims)), (0.04, 0.0, 0.0)))
        assert a.slots > 1024
        for k in range(3):
            for n in [1] * 5 if single else (5,):
                a.step(n)
            a.set_body(lbm.make_body(**dict(body, centre=(20.3 + vx * (k + 1) * 8, 20.0, 19.9))))
            a.step(1)
        runs.append(a.read_coarse() + a.read_pool() + (a.forces(), a.topology()["block_slot"]))
        a.close()
    for x, y in zip(*runs):
        assert np.array_equal(x, y)
    assert abs(runs[0][4][0]) > 0


@pytest.mark.parametrize("bounceback", [0, 1])
def test_fused_2d_macro_steps_with_more_tiles_than_blocks(lbm, bounceback):
    from getting_air_b200 import scenarios as sc
    s = sc.cylinder_amr(W=512, H=256, r=14.0, centre=(150.0, 128.0), u0=0.08, re=100.0, bounceback=bool(bounceback))
    out = []
    for fused in (True, False):
        a = lbm.Amr2D(lbm.amr2d_config(512, 256, refine_margin=100.0, **s["kw"]))
        a.set_fused(fused)
        assert a.fused == fused
        a.write_root(s["f"], s["vel"])
        a.step(5)
        a.step(16)
        a.sync()
        out.append(a.read_root() + a.read_pool() + (a.forces(), a.topology()["active"]))
        a.close()
    assert len(out[0][5]) > 2 * 148
    for x, y in zip(*out):
        assert np.array_equal(x, y)


@pytest.mark.parametrize("q,dims", [(19, (40, 24, 22)), (9, (70, 40, 1))])
def test_force_counts_nonfinite_cells(lbm, q, dims):
    """Non-finite contributions are dropped and counted, in a block's partial
    (one cell per thread) as in the batch's running sums."""
    import torch
    body = dict(shape="sphere" if q == 19 else "ellipse", a=5.0, b=5.0,
                centre=(14.0, 12.0, 11.0) if q == 19 else (30.0, 20.0, 0.0))
    cfg = lbm.config_from(q, dims, tau=0.6, body=body, **BODY)
    s, b = lbm.Solver(cfg), lbm.Batch([cfg])
    n = int(np.prod(dims))
    mac = np.tile(np.array([1.0, 0.04, 0.0, 0.0], np.float32), (n, 1))
    s.init_macro(mac)
    f = np.array(s.read_f())
    # fluid cells beside the body, whole columns of them
    x = np.arange(n) % dims[0]
    f.reshape(q, n)[:, x == (20 if q == 19 else 36)] = np.nan
    f.reshape(q, n)[:, x == (8 if q == 19 else 24)] = np.inf
    f.reshape(q, n)[:, x == (19 if q == 19 else 35)] = np.nan
    s.write_f(f)
    b.write_f(0, f)
    din = torch.tensor(f, device="cuda")
    dout, force = torch.empty_like(din), torch.zeros(8, dtype=torch.float64, device="cuda")
    lbm.step_noalloc(cfg, din.data_ptr(), dout.data_ptr(), None, force.data_ptr(),
                     torch.cuda.current_stream().cuda_stream)
    torch.cuda.synchronize()
    s.step(1)
    b.step(1)
    g, h, k = s.forces(), b.forces()[0], force.cpu().numpy()
    assert np.isfinite(g).all() and np.array_equal(g, k[:6])
    # FP64 sums of the same cell contributions, differently grouped
    assert np.allclose(g, h, rtol=1e-10, atol=1e-12 * np.abs(h).max())
    assert k[6] > 0 and k[6] == int(k[6]) and k[7] == 0
    s.close()
    b.close()
