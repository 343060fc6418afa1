"""Fragment-memory energies: as good as their rows' sums in the FP64 form, and
the same bits in both forms however the rows are spread over work units."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _reference(c):
    """The energy (fix_backbone.cpp:4079-4177) with numpy's 80-bit numbers, the
    number of Gaussians, and the sum of what half a unit in the last place of
    every distance changes them by."""
    L = np.longdouble
    seq, x = c["seq"].decode(), c["x"].astype(L)
    mca, mcb = c["mem_ca"].reshape(-1, 9, 3).astype(L), c["mem_cb"].reshape(-1, 9, 3).astype(L)
    e, count, slope = L(0), 0, 0.0
    for m in range(c["n_mem"]):
        p = int(c["mem_pos"][m])
        for a in range(6):
            for b in range(a + 3, 9):
                i, j = p + a, p + b
                var = L(j - i) ** L(0.3)
                for u, v in ((0, 0), (0, 1), (1, 0), (1, 1)):
                    if (u and seq[i] == "G") or (v and seq[j] == "G"):
                        continue
                    d = x[i, 2 * u] - x[j, 2 * v]
                    q = (mcb if u else mca)[m, a] - (mcb if v else mca)[m, b]
                    r, r0 = np.sqrt(d @ d), np.sqrt(q @ q)
                    dr = r - r0
                    g = np.exp(-dr * dr / (2 * var))
                    e -= g
                    count += 1
                    slope += float(g * abs(dr) / var * (r + r0)) * 2.0 ** -53
    return e, count, slope


@pytest.mark.parametrize("seed", range(6))
def test_energy_is_as_good_as_its_rows(seed, tmp_path, gpu_lib):
    import torch

    from awsemmd_b200 import engine, synth

    c = synth.chain_arrays(9 + seed, 7100 + seed, n_mem_per_window=1 + seed % 2)
    want, count, slope = _reference(c)
    # Each distance and each difference of distances is good to four roundings of its own size (three squares, their sum
    # and the root; the stored one alike), each Gaussian to eight units in its last place (an argument of at most a few
    # units where it counts, the function, its sum into the row), the rows' low parts to 2^-53
    tol = 4 * 2 * slope + count * 8 * 2.0 ** -53 + 6 * c["n_res"] * 2.0 ** -53 + abs(float(want)) * 2.0 ** -53
    assert tol < 1e-11  # where rounding rows to 2^-32 leaves 1e-10
    ff = synth.forcefield_dir(str(tmp_path / "ff"))
    x0 = c["x"].reshape(-1, 3)
    with engine.AwsemBatch.from_arrays(ff, [c], precision="fp64") as s:
        got = [s.compute(x0)[1][12]]
        x = torch.tensor(np.ascontiguousarray(c["x"][:, [0, 2, 1]]), device="cuda")
        f, e = torch.empty_like(x), torch.empty(1, dtype=torch.float64, device="cuda")
        fn = s.lib.awsem_fragmem_noalloc
        fn.argtypes = [C.c_void_p] * 5
        assert fn(s.h, x.data_ptr(), f.data_ptr(), e.data_ptr(), torch.cuda.current_stream().cuda_stream) == 0
        got.append(e.item())
        s.set_state(x=x0)
        s.run(0, langevin=False)
        got.append(s.energies(0)[12])
    for g in got:
        assert abs(np.longdouble(g) - want) <= tol, (g, want, tol)


@pytest.mark.parametrize("weighted", [False, True])
@pytest.mark.parametrize("prec", ["fp64", "mixed"])
def test_energy_does_not_depend_on_the_units(prec, weighted, tmp_path, gpu_lib):
    from awsemmd_b200 import engine, synth

    c = synth.chain_arrays(150, 7200, n_mem_per_window=7)
    if weighted:
        c["mem_weight"] = np.linspace(1e-6, 1.5, c["n_mem"])  # rows of the mixed form that 2^-32 does not hold
    ff = synth.forcefield_dir(str(tmp_path / "ff"))
    x0 = c["x"].reshape(-1, 3)
    got = []
    with engine.AwsemBatch.from_arrays(ff, [c], precision=prec) as s:
        got.append(s.compute(x0))
        for shapes in ((6, 148, 148, 0), (6, 148, 148, 2), (1, 148, 148, 0), (2, 148, 148, 1), (3, 148, 148, 3)):
            s.set_launch_shapes(shapes)
            got.append(s.compute(x0))
        for form in ("kernels", "persistent"):
            s.set_step_form(form)
            s.set_state(x=x0)
            rows = s.run(0, langevin=False, thermo=True)
            got.append((got[0][0], np.append(s.energies(0)[:20], 0.0)))
            assert np.array_equal(rows, s.run(0, langevin=False, thermo=True))
    for f, e in got[1:]:
        assert np.array_equal(f, got[0][0])
        assert np.array_equal(e, got[0][1])
