"""The fused two-kernel PCG, which scenes too large to be resident run on: against the per-kernel PCG
(pcg_mode 1) with both preconditioners and precisions, in a batch, and as the fallback of an oversize
scene with its kernels chosen by the autotuner."""
import numpy as np
import pytest

from mguso import ImplicitBatch, ImplicitSolver, scenes

pytestmark = pytest.mark.gpu


def coarse_sheath(width=0.5, torso_scale=0.9):
    return scenes.sheath_on_torso(edge=0.03, torso_res=(30, 29), width=width, torso_scale=torso_scale)


def stepped(ctx, sc, precision, steps, **params):
    g = ImplicitSolver(ctx, dict(sc, params=dict(sc["params"], **params)), precision)
    st = g.step(steps)
    out = g.positions.astype(np.float64), st, g.pcg_kernels()
    g.close()
    return out


def agree(a, b, start):
    """The same iteration with its dot products summed in another order: positions within the Newton
    tolerance (1e-3 of the displacement), counts close, as the step tests of the other PCGs."""
    (pa, sa, _), (pb, sb, _) = a, b
    assert np.abs(pa - pb).max() <= 1e-3 * np.abs(pb - start).max()
    for x, y in zip(sa, sb):
        assert x["status"] == 0 and y["status"] == 0
        assert abs(x["newton_iters"] - y["newton_iters"]) <= 1
        assert abs(x["max_cg_iters"] - y["max_cg_iters"]) <= max(5, y["max_cg_iters"] // 10)


@pytest.mark.parametrize("precision", ["fp32", "mixed"])
@pytest.mark.parametrize("precond", [2, 1])
def test_fused_matches_per_kernel_and_resident(ctx, precision, precond):
    sc = coarse_sheath()
    ref = stepped(ctx, sc, precision, 2, precond=precond, pcg_mode=1)
    agree(stepped(ctx, sc, precision, 2, precond=precond), ref, sc["positions"])
    for variant in (1, 8, 22):  # one-warp and three-warp domain kernels, all rows kernels but one
        got = stepped(ctx, sc, precision, 2, precond=precond, pcg_variant=variant)
        assert got[2][0] == (variant - 1) // 6
        agree(got, ref, sc["positions"])


@pytest.mark.parametrize("precision", ["fp32", "mixed"])
@pytest.mark.parametrize("precond", [2, 1])
def test_batch_on_the_fused_kernels_matches_instances_alone(ctx, precision, precond):
    scs = [coarse_sheath(w, t) for w, t in ((0.50, 0.9), (0.60, 1.02), (0.70, 1.14))]
    scs = [dict(sc, params=dict(sc["params"], precond=precond, pcg_variant=1)) for sc in scs]
    b = ImplicitBatch(ctx, scs, precision)
    bst = b.step(2)
    for k, sc in enumerate(scs):
        alone = stepped(ctx, sc, precision, 2, pcg_variant=0)
        agree((b.instance_positions(k).astype(np.float64), [s[k] for s in bst], None), alone, sc["positions"])
    b.close()


def test_oversize_scene_on_autotuned_kernels(ctx):
    sc = scenes.sheet_on_sphere(360, height=0.32, seed=360)
    got = stepped(ctx, sc, "mixed", 1, precond=1)
    assert got[2][0] >= 0  # chosen in the step: it was not resident
    agree(got, stepped(ctx, sc, "mixed", 1, precond=1, pcg_mode=1), sc["positions"])
