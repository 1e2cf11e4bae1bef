"""The real-RF form of the pSSFP simulation (csrc/pssfp_real.cuh): its three loops (second order, third
order, any angle and relaxation), odd and even RF sample counts, voxels whose transverse magnetisation does
not outlive the pulse, and that no voxel changes another's bits. Tolerance: the FP32 bound of the simulations, 1e-5 relative L2 against the FP64 oracle.
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


def _check(cb, ctx, oracle, p, seq):
    params = cb.TissueParameters.from_soa(ctx, p)
    s = cb.pSSFPSequence.from_dict(ctx, seq)
    value = cb.simulate_magnetization(ctx, params, s).to_numpy()
    assert oracle.rel_l2(value, oracle.pssfp(p, seq)) < TOL_FP32
    t = cb.simulate_magnetization_tangents(ctx, params, s)
    assert np.array_equal(t["echos"].to_numpy(), value)
    for name, field in (("T1", 0), ("T2", 1)):
        assert oracle.rel_l2(t[name].to_numpy(), oracle.derivative_central(oracle.pssfp, p, seq, field)) < TOL_FP32, name


# largest angle of one RF sample: 40° over nrf samples (0.1 rad at 15: second order), times scale
@pytest.mark.parametrize("nrf,scale", [(15, 1.0), (16, 1.0), (15, 2.5), (7, 1.0), (2, 1.0), (1, 1.0), (15, 8.0), (65, 1.0)])
@pytest.mark.parametrize("nz", [1, 2, 3, 9, 35])
def test_modes_against_oracle(cb, ctx, oracle, nrf, scale, nz):
    rng = np.random.default_rng([nrf, nz])
    seq = W.pssfp_sequence(rng, 19, nrf=nrf, nz=nz)
    seq["rf"] = (seq["rf"] * scale * rng.uniform(0.5, 1.0, 19)).astype(np.complex64)
    _check(cb, ctx, oracle, W.tissue_voxels(rng, 37, 22.4), seq)


# one sample of 20° to 360° (B1 0.8 to 1.2): across the ends of the short series (0.5 rad), the long ones (3π/2)
# and the half angle's sign
@pytest.mark.parametrize("degrees", [24.0, 28.0, 29.0, 90.0, 180.0, 225.0, 260.0, 280.0, 360.0])
@pytest.mark.parametrize("nz", [1, 9])
def test_large_angles_against_oracle(cb, ctx, oracle, degrees, nz):
    rng = np.random.default_rng([int(degrees), nz])
    seq = W.pssfp_sequence(rng, 19, nrf=1, nz=nz)
    seq["rf"] = (degrees * np.sign(seq["rf"].real)).astype(np.complex64)
    _check(cb, ctx, oracle, W.tissue_voxels(rng, 37, 22.4), seq)


def test_short_relaxation_times(cb, ctx, oracle):
    # T2 of 20 us to 1 ms beside ordinary voxels: pulses of 1 ms take up to e^-50
    rng = np.random.default_rng(3)
    seq = W.pssfp_sequence(rng, 19, nrf=15, nz=9)
    p = W.tissue_voxels(rng, 130, 22.4)
    p[1, ::7] = np.geomspace(2e-5, 1e-3, p[1, ::7].size)
    params = cb.TissueParameters.from_soa(ctx, p)
    got = cb.simulate_magnetization(ctx, params, cb.pSSFPSequence.from_dict(ctx, seq)).to_numpy()
    assert np.isfinite(got).all()
    assert oracle.rel_l2(got, oracle.pssfp(p, seq)) < TOL_FP32


@pytest.mark.parametrize("nv", [50, 1100, 6000, 20000])
def test_layout_choice_covers_voxel_counts(cb, ctx, oracle, nv):
    # few voxels take more lanes each: the same echoes to FP32 rounding whatever the choice
    rng = np.random.default_rng(4)
    seq = W.pssfp_sequence(rng, 17, nrf=5, nz=35)
    p = W.tissue_voxels(rng, nv, 22.4)
    got = cb.simulate_magnetization(ctx, cb.TissueParameters.from_soa(ctx, p), cb.pSSFPSequence.from_dict(ctx, seq))
    idx = np.arange(0, nv, max(1, nv // 40))
    assert oracle.rel_l2(got.to_numpy()[:, idx], oracle.pssfp(p, seq, vidx=idx)) < TOL_FP32


@pytest.mark.parametrize("row,bad", [(1, 0.0), (1, 1e-6), (1, np.nan), (0, 0.0), (3, 5e3), (3, np.nan), (2, 40.0), (2, np.inf)])
@pytest.mark.parametrize("nz,scale", [(1, 1.0), (9, 1.0), (35, 1.0), (9, 2.5)])
def test_a_voxel_leaves_its_neighbours_alone(cb, ctx, row, bad, nz, scale):
    # one voxel without relaxation times, with a NaN, or with large angles (off-resonance of 2 rad per RF
    # sample, 40 times the flip angle) needs more than the others of its warp: their bits stay
    rng = np.random.default_rng([nz, row])
    seq = W.pssfp_sequence(rng, 13, nrf=15, nz=nz)
    seq["rf"] = (seq["rf"] * scale).astype(np.complex64)
    s = cb.pSSFPSequence.from_dict(ctx, seq)
    nv = 45 if nz == 1 else 20001  # many voxels: several to a warp
    p = W.tissue_voxels(rng, nv, 22.4)

    def run(p):
        params = cb.TissueParameters.from_soa(ctx, p)
        t = cb.simulate_magnetization_tangents(ctx, params, s)
        return [cb.simulate_magnetization(ctx, params, s).to_numpy()] + [t[k].to_numpy() for k in ("echos", "T1", "T2")]

    ref = run(p)
    p[row, 7] = bad
    keep = np.arange(nv) != 7
    for a, b in zip(run(p), ref):
        assert np.array_equal(a[:, keep], b[:, keep])


def test_large_angles_and_masked_voxels_against_oracle(cb, ctx, oracle):
    # off-resonance of up to 1 rad per sample beside voxels on resonance and voxels with T2 = 0
    rng = np.random.default_rng(6)
    seq = W.pssfp_sequence(rng, 19, nrf=15, nz=9)
    p = W.tissue_voxels(rng, 130, 22.4)
    p[3, ::3] = rng.uniform(-2400.0, 2400.0, p[3, ::3].size)
    _check(cb, ctx, oracle, p, seq)
    p[1, 1::5] = 0.0
    got = cb.simulate_magnetization(ctx, cb.TissueParameters.from_soa(ctx, p), cb.pSSFPSequence.from_dict(ctx, seq)).to_numpy()
    assert np.array_equal(got[:, 1::5], np.zeros_like(got[:, 1::5]))
    keep = np.arange(130) % 5 != 1
    assert oracle.rel_l2(got[:, keep], oracle.pssfp(p[:, keep], seq)) < TOL_FP32


@pytest.mark.parametrize("nz", [1, 3, 5, 9, 12, 20, 35, 48, 64])
def test_batch_bits_are_those_of_each_job_alone(cb, ctx, oracle, nz):
    # a batch takes one layout for all its voxels and sums each job's isochromats in the order of the job's own
    # layout, for many or few voxels; jobs with voxels of every loop. Between the layouts only that order differs.
    rng = np.random.default_rng([8, nz])
    seq = W.pssfp_sequence(rng, 9, nrf=4, nz=nz)
    seq["gz"] = (0.09, seq["gz"][1], seq["gz"][2])
    p = W.tissue_voxels(rng, 40001, 22.4)
    p[3, ::11] = rng.uniform(-3000.0, 3000.0, p[3, ::11].size)
    p[3, 5::301] = 5000.0
    s = cb.pSSFPSequence.from_dict(ctx, seq)
    cuts = [(0, 40001), (100, 9100), (5000, 8000), (300, 1500), (200, 260), (7, 8)]
    params = [cb.TissueParameters.from_soa(ctx, np.ascontiguousarray(p[:, a:b])) for a, b in cuts]
    many = cb.simulate_magnetization(ctx, params[0], s).to_numpy()
    for jobs in (range(6), range(1, 6), (3, 5), (4, 5)):
        tangents = [i % 2 == 1 for i in jobs]
        batch = cb.SimulationBatch(ctx, [(params[i], s, None, None) for i in jobs], tangents=tangents)
        batch.run()
        ctx.synchronize()
        for n, (i, tan) in enumerate(zip(jobs, tangents)):
            alone = cb.simulate_magnetization_tangents(ctx, params[i], s) if tan else None
            echos = (alone["echos"] if tan else cb.simulate_magnetization(ctx, params[i], s)).to_numpy()
            assert np.array_equal(batch.echos(n).to_numpy(), echos), (nz, i)
            assert oracle.rel_l2(echos, many[:, cuts[i][0]:cuts[i][1]]) < 1e-6
            if tan:
                for f in ("T1", "T2"):
                    assert np.array_equal(batch.derivative(n, f).to_numpy(), alone[f].to_numpy()), (nz, i, f)
