"""Packs of four and two slices of one geometry in a batch plan's graph: 2, 3, 5, 6 and 7 slices of one
geometry each (packs of four and two and single slices side by side), in shuffled order and separate
arrays, with sizes that leave partial tiles, bins not a multiple of four, a cover subset rule, an
off-centre axis and a sinogram correction.  Against the same plan serving every slice alone (groups
off; the bound of the group tests, the order of float sums) and the oracle."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu

SS, IT = 4, 2


@pytest.mark.parametrize("counts", [(2, 2, 3), (5, 7, 1), (4, 6, 4), (2, 3, 7)])
def test_packs_match_single_slices(gpu_ctx, oracle_lib, counts):
    import xct
    from xct import phantom as P
    O = oracle_lib
    shapes = [  # nx, ny, px, angles, centre offset, cover, correction
        (403, 377, 421, 62, 1.75, True, 0),
        (349, 349, 352, 60, 0.0, False, 2),
        (292, 330, 340, 63, -2.5, False, 0),
    ]
    order = np.random.default_rng(sum(counts)).permutation([k for k, c in enumerate(counts) for _ in range(c)])
    geoms, sinos, specs = [], [], []
    for j, k in enumerate(order):
        nx, ny, px, pa, off, cover, corr = shapes[k]
        ang = P.uniform_angles(pa)
        m = max(nx, ny)
        img = P.rasterize_ellipses(P.ellipse_params(m, 6, 40 + j, axes=(2, m / 4)), m, m)[:ny, :nx].copy()
        meas = P.noisy_log_sinogram(O.projection(img, ang, px, cx=px * 0.5 + off), 1e5, j).astype(np.float32)
        mode = xct.SUBSETS_COVER if cover else xct.SUBSETS_REF
        geoms.append(xct.make_geom(nx, ny, px, ang, SS, IT, center_bin=px * 0.5 + off, subset_mode=mode,
                                   correction_mode=corr))
        sinos.append(torch.from_numpy(meas).cuda())
        specs.append((nx, ny, px * 0.5 + off, ang, cover, corr, meas))

    def run(plan):
        imgs = [torch.ones((s[1], s[0]), device="cuda") for s in specs]
        n0 = xct.launch_count()
        plan.run(sinos, imgs)
        torch.cuda.synchronize()
        return [x.cpu().numpy().astype(np.float64) for x in imgs], xct.launch_count() - n0

    bp = xct.BatchPlan(gpu_ctx, geoms, IT)
    assert bp.groups() == (0, 0)
    packed, n_packed = run(bp)
    again, _ = run(bp)
    bp.set_grouping(False)
    alone, n_alone = run(bp)
    bp.close()
    corrected = int(any(s[5] for s in specs))
    sizes = sum(any(c >> b & 1 if b < 2 else c >= 4 for c in counts) for b in range(3))
    assert n_alone == 3 * SS * IT + corrected
    assert n_packed == (2 * sizes + 1) * SS * IT + corrected
    seen = set()
    for i, k in enumerate(order):
        a, b = packed[i], alone[i]
        assert np.linalg.norm(a - b) <= 1e-6 * np.linalg.norm(b), i
        assert np.linalg.norm(again[i] - b) <= 1e-6 * np.linalg.norm(b), i
        if k not in seen:
            seen.add(k)
            nx, ny, cx, ang, cover, corr, meas = specs[i]
            used = O.sino_correction(meas, ang, corr) if corr else meas
            ref = O.osem_run(np.ones((ny, nx), np.float32), used, ang, SS, IT, cx=cx, cover=cover, order=O.ORDER_LITERAL)
            assert np.linalg.norm(a - ref) <= 1e-4 * np.linalg.norm(ref), i
            assert np.abs(a - ref).max() <= 1e-3 * np.abs(ref).max(), i
