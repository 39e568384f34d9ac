"""The library's host code over a stand-in for the CUDA runtime
(tests/native/fake_cuda.cpp): index arithmetic at sizes that no test machine
holds, and what is left behind when a call of the runtime fails."""
from __future__ import annotations

import ctypes

import numpy as np
import pytest


def _ptr(a):
    return a.ctypes.data_as(ctypes.c_void_p)


@pytest.fixture
def fake(fakecuda):
    fakecuda.fake_reset()
    yield fakecuda
    fakecuda.fake_reset()


def _train(fake, n, batch, steps, seed=9):
    """the (start, size) of every mini-batch of lbm_mlp_train"""
    P = np.zeros(fake.lbm_mlp_param_count(), np.float32)
    x = ctypes.c_void_p(16)   # never read: the kernels are stand-ins
    rc = fake.lbm_mlp_train(x, x, n, batch, steps, ctypes.c_float(1e-3), seed, _ptr(P), None, None)
    assert rc == 0, fake.lbm_last_error()
    out = (ctypes.c_longlong * (2 * steps))()
    assert fake.fake_trace(out, 2 * steps) == 2 * steps
    return [(out[2 * i], out[2 * i + 1]) for i in range(steps)]


@pytest.mark.parametrize("n,batch", [(1 << 30, 1 << 30), (1_200_000_000, 1_000_000_000), (2 ** 31 - 1, 2 ** 30)])
def test_batches_stay_inside_the_samples(fake, n, batch):
    """batches near 2^31 samples (position + batch passes the range of an
    int): each lies within the permutation"""
    for start, size in _train(fake, n, batch, 4):
        assert 0 <= start and start + size <= n


def _solver(fake, **kw):
    import lbm_multigpu_gb300 as lbm

    h = ctypes.c_void_p()
    text = lbm.make_inputs(64, 24, 12, obst1=(18.5, 11.5, 0.0), r1=4.0, re=60.0, umax=0.05, tmax=1000, les=1, cs=0.01,
                           bounceback="halfway", **kw)
    assert fake.lbm_create(text.encode(), ctypes.byref(h)) == 0, fake.lbm_last_error()
    return h


@pytest.mark.parametrize("call", ["cudaStreamBeginCapture", "cudaStreamEndCapture", "cudaGraphInstantiate"])
def test_failed_capture_leaves_no_stale_graph(fake, call):
    """a capture that fails after a mask change: the next call captures the
    steps anew instead of launching the graph of the old mask"""
    h = _solver(fake)
    mask = np.zeros((12, 24, 64), np.uint8)
    assert fake.lbm_step(h, 64) == 0
    assert fake.lbm_set_mask(h, 0, _ptr(mask)) == 0, fake.lbm_last_error()
    fake.fake_mark()
    if call == "cudaGraphInstantiate":   # reached when the old executable cannot be updated in place
        fake.fake_fail(b"cudaGraphExecUpdate", 1)
    fake.fake_fail(call.encode(), 1)
    assert fake.lbm_step(h, 64) != 0
    fake.fake_fail(b"cudaGraphExecUpdate", 0)
    launches = fake.fake_calls(b"cudaGraphLaunch")
    assert fake.lbm_step(h, 64) == 0, fake.lbm_last_error()
    assert fake.fake_calls(b"cudaGraphLaunch") > launches and fake.fake_stale_launches() == 0
    assert fake.lbm_destroy(h) == 0


@pytest.mark.parametrize("call", ["cudaMalloc", "cudaMemcpy"])
@pytest.mark.parametrize("before", [0, 1])
def test_modes_after_a_failed_initialisation(fake, call, before):
    """lbm_ensemble_modes after an lbm_ensemble_init_turbulence that failed on
    the device: the modes of the last field that was made (before: an earlier
    one with fewer modes), none without one"""
    h, sizes, tau = ctypes.c_void_p(), np.array([32, 48], np.int32), np.array([0.6, 0.6], np.float32)
    assert fake.lbm_ensemble_create(2, _ptr(sizes), _ptr(tau), 0, ctypes.c_float(0.01), ctypes.byref(h)) == 0

    def modes(member):
        n = ctypes.c_int()
        k, ph, a = np.zeros((4096, 3), np.int32), np.zeros(4096), np.zeros((4096, 3))
        assert fake.lbm_ensemble_modes(h, member, _ptr(k), _ptr(ph), _ptr(a), 4096, ctypes.byref(n)) == 0
        return n.value, k[:n.value].copy(), ph[:n.value].copy(), a[:n.value].copy()

    u = ctypes.c_float(0.04)
    if before:
        assert fake.lbm_ensemble_init_turbulence(h, 1, u, 16, 2) == 0, fake.lbm_last_error()
    want = [modes(m) for m in range(2)]
    assert (want[1][0] > 0) == bool(before)
    fake.fake_fail(call.encode(), 1)
    assert fake.lbm_ensemble_init_turbulence(h, 2, u, 4, 24) != 0
    for m in range(2):
        got = modes(m)
        assert got[0] == want[m][0]
        for x, y in zip(got[1:], want[m][1:]):
            np.testing.assert_array_equal(x, y)
    assert fake.lbm_ensemble_destroy(h) == 0


def test_closure_grid_is_of_the_device(fake):
    """the closure kernel's grid, with the function attributes that go with
    it, is worked out once on each device; a failure is not kept"""
    g = ctypes.c_int()
    assert fake.fake_device_grid(1, 1, ctypes.byref(g)) != 0
    for device in (0, 1, 0, 1, 63):
        assert fake.fake_device_grid(device, 0, ctypes.byref(g)) == 0 and g.value == 100 * (device + 1)
    assert fake.fake_calls(b"grid") == 4
    assert fake.fake_device_grid(64, 0, ctypes.byref(g)) != 0


@pytest.mark.parametrize("calls,captures", [([5, 20], 0), ([4, 4, 4], 0), ([8, 8, 8], 1), ([20, 20, 20], 2),
                                            ([20, 640], 1), ([100], 1)])
def test_short_calls_capture_nothing_they_do_not_use_again(fake, calls, captures):
    """a batch is captured when one of its kind comes a second time: a first
    short call is direct steps, and what is captured is launched again"""
    h = _solver(fake)
    for n in calls:
        assert fake.lbm_step(h, n) == 0, fake.lbm_last_error()
    assert fake.fake_calls(b"cudaStreamBeginCapture") == captures
    assert fake.fake_calls(b"cudaGraphLaunch") >= captures
    assert fake.lbm_destroy(h) == 0


@pytest.mark.parametrize("n,epochs,room", [(1, 3, True), (2, 3, True), (4000, 3, True), (28_671, 2, True),
                                           (28_672, 2, False), (100_003, 2, False)])
def test_host_shuffle(fake, n, epochs, room):
    """with few samples, or without device memory for the device's shuffle,
    training shuffles on the host, in the order of the oracle's shuffle"""
    from oracle_bindings import oracle

    if not room:
        fake.fake_fail_above(b"cudaMallocFromPoolAsync", ctypes.c_size_t(8 * n))
    batch, P, x = (n + 1) // 2, np.zeros(fake.lbm_mlp_param_count(), np.float32), ctypes.c_void_p(16)
    per = n // batch   # steps an epoch
    blocks = fake.fake_blocks()
    assert fake.lbm_mlp_train(x, x, n, batch, per * epochs, ctypes.c_float(1e-3), 9, _ptr(P), None, None) == 0
    assert fake.fake_calls(b"launch_shuffle") == 0 and fake.fake_blocks() == blocks
    got = np.zeros(per * epochs * batch, np.int64)
    assert fake.fake_trace(_ptr(got), len(got)) == len(got)
    shuffle = oracle().orc_shuffle
    shuffle.restype, shuffle.argtypes = ctypes.c_uint64, [ctypes.c_uint64, ctypes.c_void_p, ctypes.c_int]
    state, perm, want = (9 * 0x9E3779B97F4A7C15 + 0x632BE59BD9B4E019) % 2 ** 64, np.arange(n, dtype=np.int32), []
    for _ in range(epochs):
        state = shuffle(state, _ptr(perm), n)
        want.append(perm[:per * batch].copy())
    np.testing.assert_array_equal(got, np.concatenate(want))


def test_device_shuffle_from_its_size_on(fake):
    """the rule's other side: with room for its scratch the shuffle of 28,672
    samples is the device's"""
    _train(fake, 28_672, 28_672, 3)
    assert fake.fake_calls(b"launch_shuffle") == 3


@pytest.mark.parametrize("nx,ny,nz", [(31, 13, 5), (33, 12, 6), (64, 12, 5), (70, 24, 6)])
def test_statistics_without_staging_memory(fake, nx, ny, nz):
    """lbm_get_stats where the device has no room for the packed copy: row by
    row, without the padding"""
    import lbm_multigpu_gb300 as lbm

    h, pitch = ctypes.c_void_p(), (nx + 31) // 32 * 32
    text = lbm.make_inputs(nx, ny, nz, obst1=(8.5, 5.5, 0.0), r1=2.0, re=60.0, umax=0.05, tmax=10, les=1, cs=0.01,
                           geometry="channel_square", velav=1, start_velav=0, start_velfluc=5)
    assert fake.lbm_create(text.encode(), ctypes.byref(h)) == 0, fake.lbm_last_error()
    assert fake.lbm_step(h, 1) == 0
    got = np.full((4, nz, ny, nx), -1, np.float32)
    fake.fake_fail(b"cudaMalloc", 1)
    assert fake.lbm_get_stats(h, 0, _ptr(got)) == 0, fake.lbm_last_error()
    assert fake.fake_calls(b"cudaMemcpy2DAsync") == 4
    np.testing.assert_array_equal(got, np.arange(4 * nz * ny * pitch).reshape(4, nz, ny, pitch)[..., :nx])
    fake.fake_fail(b"cudaMalloc", 1)
    fake.fake_fail(b"cudaMemcpy2DAsync", 3)
    assert fake.lbm_get_stats(h, 0, _ptr(got)) != 0
    assert fake.lbm_destroy(h) == 0


@pytest.mark.parametrize("refined,calls,captures", [(0, [24], 1), (0, [20], 0), (0, [16, 16], 1), (1, [20], 1), (1, [8], 0),
                                                    (1, [20, 20], 2)])
def test_captures_of_large_domains_hide_behind_direct_steps(fake, refined, calls, captures):
    """from 4 MB a population on the first long call captures behind eight
    direct steps (with refinement four, the graph of 8), and every step is run"""
    import lbm_multigpu_gb300 as lbm

    h, kw = ctypes.c_void_p(), {}
    if refined:
        kw = dict(refinement=1, lr_dims=(64, 48, 32), lr_factor=0.5, lr_origin=(48.25, 20.25, 16.25))
    text = lbm.make_inputs(256, 64, 64, obst1=(64.5, 31.5, 0.0), r1=4.0, re=60.0, umax=0.05, tmax=1000, les=1, cs=0.01, **kw)
    assert fake.lbm_create(text.encode(), ctypes.byref(h)) == 0, fake.lbm_last_error()
    for n in calls:
        assert fake.lbm_step(h, n) == 0, fake.lbm_last_error()
    t = ctypes.c_int()
    assert fake.lbm_get_time(h, ctypes.byref(t)) == 0 and t.value == sum(calls)
    assert fake.fake_calls(b"cudaStreamBeginCapture") == captures
    assert fake.lbm_destroy(h) == 0


@pytest.mark.parametrize("dims", [(64, 24, 6), (33, 7, 5), (31, 5, 3), (70, 9, 4)])
@pytest.mark.parametrize("bounceback", ["halfway", "fullway"])
@pytest.mark.parametrize("edge", ["wrap", "clamp"])
@pytest.mark.parametrize("what", ["walls", "sparse", "body", "none"])
def test_uploaded_mask_against_brute_force(fake, dims, bounceback, edge, what):
    """the flag of nodes next to a solid one, their links, and the force list
    with its links to the body, against a look at all 18 neighbours"""
    import lbm_multigpu_gb300 as lbm
    from oracle_bindings import CX, CY, CZ

    nx, ny, nz = dims
    N, rng = lbm.NODE, np.random.default_rng(nx)
    m = np.zeros((nz, ny, nx), np.uint8)
    if what == "walls":      # at both ends of every row
        m[:, :, 0] = m[:, :, -1] = N["WALL"]
        m[nz // 2, ny // 2, nx // 2] = N["BODY"]
    elif what == "sparse":
        r = rng.random(m.shape)
        m[r < 0.02], m[r > 0.98], m[(r > 0.5) & (r < 0.52)] = N["WALL"], N["BODY"], N["WEST_INLET"]
    elif what == "body":
        m[1:3, 2:4, 5:9] = N["BODY"]
    h, pitch = ctypes.c_void_p(), (nx + 31) // 32 * 32
    text = lbm.make_inputs(nx, ny, nz, obst1=(8.5, 2.5, 0.0), r1=1.0, re=60.0, umax=0.05, tmax=10, les=1, cs=0.01,
                           bounceback=bounceback, edge_pull=edge)
    assert fake.lbm_create(text.encode(), ctypes.byref(h)) == 0, fake.lbm_last_error()
    assert fake.lbm_set_mask(h, 0, _ptr(m)) == 0 and fake.lbm_step(h, 2) == 0, fake.lbm_last_error()
    solid, body = np.isin(m, [N["WALL"], N["BODY"]]), m == N["BODY"]
    links, blinks = np.zeros(m.shape, np.uint32), np.zeros(m.shape, np.uint32)
    ax = [np.arange(n) for n in (nz, ny, nx)]
    take = (lambda i, n: np.clip(i, 0, n - 1)) if edge == "clamp" else (lambda i, n: i % n)
    for q in range(1, 19):
        at = np.ix_(take(ax[0] - int(CZ[q]), nz), take(ax[1] - int(CY[q]), ny), take(ax[2] - int(CX[q]), nx))
        links |= (solid[at] & ~solid).astype(np.uint32) << q
        blinks |= (body[at] & ~solid).astype(np.uint32) << q
    got = np.zeros((nz, ny, pitch), np.uint8)
    assert fake.fake_mask(_ptr(got)) == got.size
    np.testing.assert_array_equal(got[..., :nx], m | np.where(links != 0, 0x80, 0).astype(np.uint8))
    assert (got[..., nx:] == N["WALL"]).all()

    def words(which):
        n = fake.fake_words(which, None, 0)
        w = np.zeros(n, np.uint32)
        fake.fake_words(which, _ptr(w), n)
        return w

    if bounceback == "halfway":
        np.testing.assert_array_equal(words(0).reshape(nz, ny, pitch)[..., :nx], links)
        assert not words(0).reshape(nz, ny, pitch)[..., nx:].any()
        listed = blinks != 0
        np.testing.assert_array_equal(words(2), blinks[listed])
    else:
        listed = body
        assert words(2).size == 0
    at = np.zeros((nz, ny, pitch), np.uint32)
    at.reshape(-1)[:] = np.arange(at.size)
    np.testing.assert_array_equal(words(1), at[..., :nx][listed])
    assert fake.lbm_destroy(h) == 0


@pytest.mark.parametrize("bounceback", ["halfway", "fullway"])
@pytest.mark.parametrize("nth", [1, 2, 3])
def test_failed_mask_upload_leaves_no_half_force_list(fake, bounceback, nth):
    """lbm_set_mask that fails in one of its allocations: no later step
    reduces a force over a list that is not on the device, or over one without
    its links"""
    h, mask = ctypes.c_void_p(), np.zeros((12, 24, 64), np.uint8)
    import lbm_multigpu_gb300 as lbm

    text = lbm.make_inputs(64, 24, 12, obst1=(18.5, 11.5, 0.0), r1=4.0, re=60.0, umax=0.05, tmax=1000, les=1, cs=0.01,
                           bounceback=bounceback)
    assert fake.lbm_create(text.encode(), ctypes.byref(h)) == 0 and fake.lbm_step(h, 3) == 0
    mask[3:5, 6:9, 20:24] = lbm.NODE["BODY"]
    fake.fake_fail(b"cudaMalloc", nth)
    allocations = {"halfway": 3, "fullway": 1}[bounceback]
    assert (fake.lbm_set_mask(h, 0, _ptr(mask)) != 0) == (nth <= allocations)
    launches = fake.fake_calls(b"launch_force")
    fake.lbm_step(h, 2)
    if fake.fake_calls(b"launch_force") > launches:   # both parts of the list are there
        assert fake.fake_words(1, None, 0) > 0
        assert (fake.fake_words(2, None, 0) > 0) == (bounceback == "halfway")
    assert fake.fake_calls(b"null body list") == 0
    assert fake.lbm_destroy(h) == 0
