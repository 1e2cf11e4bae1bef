"""The real-phase form of the FISP simulation (csrc/fisp_real.cuh): sequences whose RF train and slice
profiles are real run on real states without the off-resonance phases, one layout per state count,
over 4 lanes when there are few (voxel, position) pairs. Sizes at the layouts' edges: state counts
around the pair and lane boundaries, TRs around the 64-TR (32-TR) sample chunks, ragged voxel counts.
Tolerance: the FP32 bound of the simulations, 1e-5 relative L2 against the FP64 oracle.
"""
import numpy as np
import pytest

import workloads as W

pytestmark = pytest.mark.gpu

TOL_FP32 = 1e-5


@pytest.fixture(scope="module")
def cb():
    import compas_b200

    compas_b200.library()
    return compas_b200


@pytest.fixture(scope="module")
def ctx(cb):
    return cb.Context(0)


def _case(nv, ntr, P, N, seed=1, **flags):
    rng = np.random.default_rng([seed, N, P])
    p = W.tissue_voxels(rng, nv, 22.4)
    rf = W.smooth_flip_train(rng, ntr) * np.where(rng.uniform(size=ntr) < 0.3, -1.0, 1.0)  # phases 0 and π
    rf[ntr // 2] = 0.0
    slices = rng.uniform(0.2, 1.0, (P, ntr)) * np.where(rng.uniform(size=(P, 1)) < 0.3, -1.0, 1.0)
    seq = W.fisp_sequence(rf, slices, 8.7e-3, 4.35e-3, 25e-3, N)
    seq.update(flags)
    return p, seq


def _run(cb, ctx, p, seq):
    params = cb.TissueParameters.from_soa(ctx, p)
    s = cb.FispSequence.from_dict(ctx, seq)
    t = cb.simulate_magnetization_tangents(ctx, params, s)
    return [cb.simulate_magnetization(ctx, params, s).to_numpy()] + [t[k].to_numpy() for k in ("echos", "T1", "T2")]


@pytest.mark.parametrize("N", [2, 3, 4, 5, 8, 9, 10, 13, 14, 16, 17, 18, 21, 22, 24, 25, 26, 32, 33, 34])
@pytest.mark.parametrize("nv,ntr,P", [(37, 66, 3), (1, 64, 1), (33, 33, 1)])
def test_state_counts_against_oracle(cb, ctx, oracle, N, nv, ntr, P):
    p, seq = _case(nv, ntr, P, N)
    value, echos, d1, d2 = _run(cb, ctx, p, seq)
    assert oracle.rel_l2(value, oracle.fisp(p, seq)) < TOL_FP32
    assert np.array_equal(value, echos) or N > 33  # 34 states: the general layouts
    for got, field in ((d1, 0), (d2, 1)):
        assert oracle.rel_l2(got, oracle.derivative_central(oracle.fisp, p, seq, field)) < TOL_FP32, field


@pytest.mark.parametrize("flags", [dict(reps=3, TW=0.05, uf=2), dict(reps=2, TW=0.04, wait_spoil=0),
                                   dict(reps=2, TW=0.04, inversion=0), dict(reps=2, TW=0.0, inversion=0, wait_spoil=0),
                                   dict(reps=2, TW=0.04, inversion=0, wait_spoil=0)])
@pytest.mark.parametrize("N", [6, 25])
def test_repetitions_and_flags_against_oracle(cb, ctx, oracle, N, flags):
    # the last combination precesses over the wait with transverse states alive: the general form
    p, seq = _case(35, 41, 4, N, seed=2, **flags)
    value, echos, d1, d2 = _run(cb, ctx, p, seq)
    assert oracle.rel_l2(value, oracle.fisp(p, seq)) < TOL_FP32
    assert oracle.rel_l2(echos, value) < 1e-6
    for got, field in ((d1, 0), (d2, 1)):
        assert oracle.rel_l2(got, oracle.derivative_central(oracle.fisp, p, seq, field)) < TOL_FP32, field


# transverse states that live through the wait: the packed layouts' real-phase form (enough pairs for one lane
# per voxel), alone and in a batch, beside complex phases on the general form
@pytest.mark.parametrize("N", [8, 25, 32])
def test_unspoiled_wait_on_packed_layouts(cb, ctx, oracle, N):
    p, seq = _case(2500, 21, 16, N, seed=8, reps=2, TW=0.04, inversion=0, wait_spoil=0)
    turned = dict(seq, rf=(seq["rf"] * np.exp(0.3j)).astype(np.complex64))
    idx = np.arange(0, 2500, 60)
    for s in (seq, turned):
        got = _run(cb, ctx, p, s)
        assert oracle.rel_l2(got[0][:, idx], oracle.fisp(p, s, vidx=idx)) < TOL_FP32
        for d, field in ((got[2], 0), (got[3], 1)):
            assert oracle.rel_l2(d[:, idx], oracle.derivative_central(oracle.fisp, p, s, field, vidx=idx)) < TOL_FP32
        params, sequence = cb.TissueParameters.from_soa(ctx, p), cb.FispSequence.from_dict(ctx, s)
        batch = cb.SimulationBatch(ctx, [(params, sequence, None, None)] * 2, tangents=[False, True])
        batch.run()
        ctx.synchronize()
        assert np.array_equal(batch.echos(0).to_numpy(), got[0])
        assert np.array_equal(batch.echos(1).to_numpy(), got[1])
        assert np.array_equal(batch.derivative(1, "T1").to_numpy(), got[2])


# an explicit layout override means a layout of the general kernels, for real phases too: other bits than
# the real-state kernels' (both within FP32 of each other), the same alone and in a batch
@pytest.mark.parametrize("tangents", [False, True])
def test_layout_override_runs_the_general_layout(cb, ctx, oracle, tangents):
    p, seq = _case(300, 50, 2, 8, seed=9)
    params, s = cb.TissueParameters.from_soa(ctx, p), cb.FispSequence.from_dict(ctx, seq)

    def run():
        if not tangents:
            return [cb.simulate_magnetization(ctx, params, s).to_numpy()]
        t = cb.simulate_magnetization_tangents(ctx, params, s)
        return [t[k].to_numpy() for k in ("echos", "T1", "T2")]

    force = cb.set_fisp_tangent_launch if tangents else cb.set_fisp_launch
    configs = cb.fisp_tangent_configs() if tangents else cb.fisp_configs()
    own = run()
    try:
        force(next(i for i, c in enumerate(configs) if tuple(c) == (8, 1)))
        forced = run()
        batch = cb.SimulationBatch(ctx, [(params, s, None, None)], tangents=[tangents])
        batch.run()
        ctx.synchronize()
        assert np.array_equal(batch.echos(0).to_numpy(), forced[0])
        force(next(i for i, c in enumerate(configs) if c[0] * c[1] < 8))  # does not hold the states
        small = run()
    finally:
        force(-1)
    for a, b, c in zip(own, forced, small):
        assert not np.array_equal(a, b) and oracle.rel_l2(b, a) < TOL_FP32
        assert np.array_equal(a, c)


@pytest.mark.parametrize("N,P,nv", [(8, 1, 15001), (25, 1, 15001), (13, 3, 10007), (25, 9, 10007), (4, 35, 10007)])
def test_bits_do_not_depend_on_the_layout(cb, ctx, N, P, nv):
    # one lane per voxel, whole tiles or the balanced split for many pairs, 4 lanes for a few of the same voxels
    p, seq = _case(nv, 70, P, N, seed=3)
    many = _run(cb, ctx, p, seq)
    few = _run(cb, ctx, np.ascontiguousarray(p[:, 100:141]), seq)
    for a, b, what in zip(many, few, ("value", "echos", "T1", "T2")):
        assert np.array_equal(a[:, 100:141], b), what


# angles past the range in which the fast sine and cosine are bounded (π), and trains whose errors of one
# sign add up over 1000 TRs
@pytest.mark.parametrize("train", ["5", "150", "180", "270", "360", "150-360", "5 alternating"])
def test_flip_angles_against_oracle(cb, ctx, oracle, train):
    p, seq = _case(37, 1000, 1, 25, seed=6)
    lo, hi = (float(x) for x in (train.split()[0].split("-") * 2)[:2])
    rf = np.random.default_rng(7).uniform(lo, hi, 1000)
    if train.endswith("alternating"):
        rf[1::2] *= -1
    seq.update(rf=rf.astype(np.complex64), slices=np.ones((1, 1000), np.complex64))
    value, echos, d1, d2 = _run(cb, ctx, p, seq)
    assert oracle.rel_l2(value, oracle.fisp(p, seq)) < TOL_FP32
    for got, field in ((d1, 0), (d2, 1)):
        assert oracle.rel_l2(got, oracle.derivative_central(oracle.fisp, p, seq, field)) < TOL_FP32, field


# shares of one to two tiles per CTA of the balanced split, whose tail and head fall into one round of
# warps (12 for 25 states, 16 for 4), beside the work queue of a batch, which runs whole tiles
@pytest.mark.parametrize("N,P,nv", [(25, 35, 6560), (25, 35, 8000), (25, 16, 9000), (4, 9, 14001), (4, 35, 8001)])
def test_balanced_shares_below_two_tiles_match_the_queue_bits(cb, ctx, N, P, nv):
    p, seq = _case(nv, 70, P, N, seed=5)
    params, s = cb.TissueParameters.from_soa(ctx, p), cb.FispSequence.from_dict(ctx, seq)
    batch = cb.SimulationBatch(ctx, [(params, s, None, None)])
    batch.run()
    ctx.synchronize()
    assert np.array_equal(cb.simulate_magnetization(ctx, params, s).to_numpy(), batch.echos(0).to_numpy())
    ctx.synchronize()  # no wait gave up


def test_a_voxel_without_relaxation_times_stays_alone(cb, ctx):
    # a masked voxel (T1 = T2 = 0) is as it was in the general form: finite, and no other voxel changes
    p, seq = _case(40, 40, 2, 25, seed=4)
    ref = _run(cb, ctx, p, seq)[0]
    p[0:2, 7] = 0.0
    got = _run(cb, ctx, p, seq)[0]
    assert np.isfinite(got).all()
    keep = np.arange(40) != 7
    assert np.array_equal(got[:, keep], ref[:, keep])


# ------------------------------------------------------------------------------------------------
# one launch per simulation once the host knows a sequence's form (csrc/runtime.cu, HostFlag)
# ------------------------------------------------------------------------------------------------

def _sequence(cb, ctx, kind, turned):
    turn = np.exp(0.4j) if turned else 1.0
    if kind == "fisp":
        seq = W.fisp_sequence(np.linspace(5, 60, 9) * turn, np.ones((1, 9)), 8.7e-3, 4.35e-3, 25e-3, 6)
        return cb.FispSequence.from_dict(ctx, seq)
    seq = W.pssfp_sequence(np.random.default_rng(3), 9, nrf=3, nz=2)
    seq["rf"] = (seq["rf"] * turn).astype(np.complex64)
    return cb.pSSFPSequence.from_dict(ctx, seq)


@pytest.mark.parametrize("kind", ["fisp", "pssfp"])
@pytest.mark.parametrize("turned", [False, True])
@pytest.mark.parametrize("tangents", [False, True])
def test_one_launch_once_the_form_is_known(cb, ctx, kind, turned, tangents):
    params = cb.TissueParameters.from_soa(ctx, W.tissue_voxels(np.random.default_rng(2), 70, 22.4))
    s = _sequence(cb, ctx, kind, turned)

    def run():
        if not tangents:
            return cb.simulate_magnetization(ctx, params, s).to_numpy()
        return np.stack([a.to_numpy() for a in cb.simulate_magnetization_tangents(ctx, params, s).values()])

    first = run()
    before = cb.launch_count()
    again = run()
    assert cb.launch_count() - before == 1
    assert np.array_equal(first, again)


def test_more_sequences_than_flags_and_reused_flags(cb, ctx):
    # 1100 sequences at a time of both forms in turn, then as many others on the words they gave back
    params = cb.TissueParameters.from_soa(ctx, W.tissue_voxels(np.random.default_rng(2), 33, 22.4))
    ref = [cb.simulate_magnetization(ctx, params, _sequence(cb, ctx, "fisp", t)).to_numpy() for t in (False, True)]
    for shift in (0, 1):
        kept = [_sequence(cb, ctx, "fisp", (i + shift) % 2 == 1) for i in range(1100)]
        for _ in range(2):
            got = [cb.simulate_magnetization(ctx, params, s) for s in kept]
            for i, g in enumerate(got):
                assert np.array_equal(g.to_numpy(), ref[(i + shift) % 2]), i
        del kept, got


@pytest.mark.parametrize("kind", ["fisp", "pssfp"])
@pytest.mark.parametrize("turned", [False, True])
def test_threads_that_share_a_new_sequence(cb, ctx, kind, turned):
    # the first calls, which do not know the form yet, and later ones from four threads at once
    from concurrent.futures import ThreadPoolExecutor

    params = cb.TissueParameters.from_soa(ctx, W.tissue_voxels(np.random.default_rng(2), 70, 22.4))
    ref = cb.simulate_magnetization(ctx, params, _sequence(cb, ctx, kind, turned)).to_numpy()
    s = _sequence(cb, ctx, kind, turned)
    with ThreadPoolExecutor(4) as pool:
        for got in pool.map(lambda _: cb.simulate_magnetization(ctx, params, s).to_numpy(), range(200)):
            assert np.array_equal(got, ref)
