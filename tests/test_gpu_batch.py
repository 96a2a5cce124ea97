"""Batched screening (ptg_batch_*): several structures in one persistent launch
replayed as a CUDA graph.  Each geometry must get exactly the counts of its
own ptg_kappa run with the same particles, seed and stream (integer tallies:
exact), and the same kappa (1e-12); replaying the graph gives the same
result again."""
import numpy as np
import pytest

from ptrans_b200 import abi as A
from ptrans_b200 import synth

pytestmark = pytest.mark.gpu


def test_batch_equals_individual_runs():
    models, _ = synth.film_batch(n=6, seed=3, n_modes=40, nangle=9)
    nps = [17, 300, 5, 120, 64, 1]
    seeds = [1, 2, 3, 4, 5, 6]
    streams = [0, 7, 0, 3, 11, 2]
    spec = synth.spectrum(40, seed=1)
    bins = (0.0, float(spec.omega.max()))
    bufs = [A.GeomBuf(m) for m in models]
    run = A.make_run(kind_mfp=A.MFP_PER_MODE, nangle=9, np_=1, nbins=8, bin_omega=bins)
    with A.Batch([b.view for b in bufs], nps, seeds, streams, spec, run) as bt:
        r1 = bt.run(want_counts=True)
        r2 = bt.run(want_counts=True)
    np.testing.assert_array_equal(r1["counts"], r2["counts"])
    np.testing.assert_array_equal(r1["kappa"], r2["kappa"])
    for g in range(len(models)):
        single = A.make_run(kind_mfp=A.MFP_PER_MODE, nangle=9, np_=nps[g], seed=seeds[g],
                            stream=streams[g], nbins=8, bin_omega=bins)
        with A.Handle(bufs[g].view, spec) as h:
            k = h.kappa(single, want_counts=True)
        np.testing.assert_array_equal(r1["counts"][g], k["counts"])
        assert r1["kappa"][g] == pytest.approx(k["kappa"], rel=1e-12)
        assert r1["kappa_stderr"][g] == pytest.approx(k["kappa_stderr"], rel=1e-10)
        np.testing.assert_allclose(r1["bin_T"][g], k["bin_T"], rtol=1e-12, atol=1e-15)
    assert r1["samples"] == sum(nps) * 40 * 8
    assert r1["lost"] == 0


def test_batch_adjoint_equals_individual_adjoints():
    """ptg_batch_adjoint gives every geometry what ptg_adjoint gives for its
    own run: the same kappa (the same counts), the same replayed samples, the
    same specularity derivatives up to the order of the FP64 sums (the scores
    of the same samples, added in another order), and the scale derivative up
    to the FP32 summation order of the samples' path lengths."""
    import dataclasses
    models, _ = synth.film_batch(n=4, seed=5, n_modes=12, nangle=7)
    models = [dataclasses.replace(m, tt_spec=np.array([0.4, 0.0]), cellspec=(1.0, 1.0, 1.0, 1.0, 0.5, 0.3))
              for m in models]
    nps = [200, 50, 400, 10]
    seeds = [11, 12, 13, 14]
    streams = [0, 3, 1, 0]
    spec = synth.spectrum(12, seed=2)
    bins = (0.0, float(spec.omega.max()))
    bufs = [A.GeomBuf(m) for m in models]
    run = A.make_run(kind_mfp=A.MFP_PER_MODE, nangle=7, np_=1, nbins=4, bin_omega=bins, precision=A.PREC_FP32)
    with A.Batch([b.view for b in bufs], nps, seeds, streams, spec, run) as bt:
        ba = bt.adjoint()
        fwd = bt.run()
    assert ba["mismatched"] == 0
    # the same counts; host (adjoint) and device (forward) FP64 assembly differ in rounding only
    np.testing.assert_allclose(ba["kappa"], fwd["kappa"], rtol=1e-12)
    replayed = 0
    for g in range(len(models)):
        single = A.make_run(kind_mfp=A.MFP_PER_MODE, nangle=7, np_=nps[g], seed=seeds[g], stream=streams[g],
                            nbins=4, bin_omega=bins, precision=A.PREC_FP32)
        with A.Handle(bufs[g].view, spec) as h:
            sa = h.adjoint(single)
        replayed += sa["replayed"]
        assert ba["kappa"][g] == pytest.approx(sa["kappa"], rel=1e-12)
        assert ba["kappa_stderr"][g] == pytest.approx(sa["kappa_stderr"], rel=1e-10)
        got, want, se = ba["dk_dp"][g], sa["dk_dp"], sa["dk_dp_stderr"]
        np.testing.assert_array_equal(np.isnan(got), np.isnan(want))
        ok = ~np.isnan(want)
        assert ok.sum() >= 3
        assert np.all(np.abs(got[ok] - want[ok]) <= 1e-6 * se[ok] + 1e-12 * np.abs(want[ok]))
        np.testing.assert_allclose(ba["dk_dp_stderr"][g][ok], se[ok], rtol=1e-6)
        # the scale score sums each sample's FP32 path length, in another order
        # where the single run's tail phase adds a round's flights by warp shuffles
        assert abs(ba["dk_dscale"][g] - sa["dk_dscale"]) <= 1e-3 * sa["dk_dscale_stderr"] + 1e-5 * abs(sa["dk_dscale"])
    assert ba["replayed"] == replayed


@pytest.mark.parametrize("kind", ["films", "bvh"])
@pytest.mark.parametrize("cap", [0, 40])
def test_batched_tail_phase_takes_the_same_trajectories(kind, cap):
    """A batch hands its last phonons to a tail phase whose warps switch
    geometry from phonon to phonon; without it (tune_flags bit 1) every phonon
    ends on one lane.  Counts, flights and lost phonons are equal, and so is
    the replayed sample set of the adjoint, in films and where several
    geometries with the same grain numbers keep a BVH and local lists."""
    if kind == "films":
        models, nps = synth.film_batch(7, seed=4, n_modes=12, nangle=5, samples_lo=500, samples_hi=9000)
    else:
        models = [synth.cube_lattice(n=n, l=300.0, fill=f, trans=0.3, spec=0.2, p_wall=0.3)
                  for n, f in ((3, 0.5), (4, 0.4), (3, 0.3))]
        models.append(synth.spheres_cylinders_box(n_spheres=4, n_cylinders=5, l=300.0, seed=3, r_sphere=(15.0, 35.0),
                                                  r_cylinder=20.0, length=(50.0, 150.0), trans=0.3, p_wall=0.2))
        nps = [37, 90, 61, 44]
    spec = synth.spectrum(12, seed=5, mfp_lo=1e-9, mfp_hi=1e-7)
    bufs = [A.GeomBuf(m) for m in models]
    run = A.make_run(kind_mfp=A.MFP_PER_MODE, nangle=5, np_=1)
    got = []
    for flags in (2, 0):
        with A.Batch([b.view for b in bufs], nps, [9 + i for i in range(len(bufs))], [0] * len(bufs), spec, run,
                     max_flights=cap, tune_flags=flags) as bt:
            r = bt.run(want_counts=True)
            again = bt.run(want_counts=True)
            a = bt.adjoint()
        np.testing.assert_array_equal(again["counts"], r["counts"])
        got.append((r["counts"], r["flights"], r["lost"], r["samples"], a["replayed"], a["mismatched"], a["flights"]))
    np.testing.assert_array_equal(got[1][0], got[0][0])
    assert got[1][1:] == got[0][1:]
    assert got[0][5] == 0


def _unlike():
    """A porous film, a convex mesh with a BVH and facet planes, capped
    cylinders and a cube lattice with a BVH alone."""
    return [synth.film_with_holes(nholes=2, seed=4, p_hole=0.5, p_z=0.3),
            synth.voronoi_box(4, box=(300.0, 250.0, 250.0), seed=5, trans=0.5, p_wall=0.3, tri_levels=2),
            synth.spheres_cylinders_box(n_spheres=4, n_cylinders=5, l=300.0, seed=3, r_sphere=(15.0, 35.0),
                                        r_cylinder=20.0, length=(50.0, 150.0), trans=0.3, p_wall=0.2),
            synth.cube_lattice(n=4, l=300.0, fill=0.4, trans=0.3, spec=0.2, p_wall=0.3)]


def test_batched_scale_derivative_does_not_depend_on_the_tail_phase():
    """A replayed sample's path length is one running sum, whichever phase flies
    it: the derivatives with and without a tail phase (tune_flags bit 1) differ
    by the order of the FP64 sums over samples alone.  Each score is below 1e3
    standard errors, so 1e-10 of the error leaves room for 1e3 roundings."""
    spec = synth.spectrum(12, seed=5, mfp_lo=1e-9, mfp_hi=1e-7)
    bufs = [A.GeomBuf(m) for m in _unlike()]
    nps, n = [37, 90, 44, 61], len(bufs)
    run = A.make_run(kind_mfp=A.MFP_PER_MODE, nangle=5, np_=1)
    got = []
    for flags in (2, 0):
        with A.Batch([b.view for b in bufs], nps, [9 + i for i in range(n)], [0] * n, spec, run,
                     tune_flags=flags) as bt:
            got.append(bt.adjoint())
    se = got[0]["dk_dscale_stderr"]
    assert np.all(se > 0.0)
    assert np.all(np.abs(got[1]["dk_dscale"] - got[0]["dk_dscale"]) <= 1e-10 * se)
    np.testing.assert_allclose(got[1]["dk_dscale_stderr"], se, rtol=1e-10)


@pytest.mark.parametrize("mfp", [(1e-9, 3e-8), (2e-8, 2e-6), None])
def test_batch_with_facet_planes_equals_linear_scans(mfp):
    """A convex mesh sends the whole batch to the kernels that use facet planes,
    the film, the capped cylinders and the lattice with it: every structure gets
    the counts of its own run without BVH and planes."""
    spec = synth.spectrum(10, seed=6, mfp_lo=mfp[0], mfp_hi=mfp[1]) if mfp else synth.spectrum(10, seed=6)
    kind = A.MFP_PER_MODE if mfp else A.MFP_MATTHIESSEN
    bufs = [A.GeomBuf(m) for m in _unlike()]
    nps, n = [37, 90, 44, 61], len(bufs)
    run = A.make_run(kind_mfp=kind, nangle=5, np_=1)
    with A.Batch([b.view for b in bufs], nps, [9 + i for i in range(n)], [0] * n, spec, run) as bt:
        r = bt.run(want_counts=True)
        replayed = bt.adjoint()["replayed"]
    for g in range(n):
        single = A.make_run(kind_mfp=kind, nangle=5, np_=nps[g], seed=9 + g)
        with A.Handle(bufs[g].view, spec, bvh_leaf=-1) as h:
            k = h.kappa(single, want_counts=True)
        np.testing.assert_array_equal(r["counts"][g], k["counts"])
        replayed -= int(k["counts"].sum())
    assert replayed == 0
