"""Fragment-memory rows at the lengths where their kernels change form: FP64
pieces of 32 records (one warp or a block a row, up to 128 records), FP32 warp
pairs; against the sums in 64 bits with numpy."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _reference(c):
    """Forces [n][CA, O, CB][3] and energy of the fragment-memory term
    (fix_backbone.cpp:4079-4177) in 64 bits."""
    n, x = c["n_res"], c["x"]
    ca, cb = x[:, 0], x[:, 2]
    seq = c["seq"].decode()
    f, e = np.zeros((n, 3, 3)), 0.0
    mca, mcb = c["mem_ca"].reshape(-1, 9, 3), c["mem_cb"].reshape(-1, 9, 3)
    for m in range(c["n_mem"]):
        p = int(c["mem_pos"][m])
        for a in range(6):
            for b in range(a + 3, 9):
                i, j = p + a, p + b
                var = float(j - i) ** 0.3
                for u, v in ((0, 0), (0, 2), (2, 0), (2, 2)):
                    if (u and seq[i] == "G") or (v and seq[j] == "G"):
                        continue
                    d = (cb if u else ca)[i] - (cb if v else ca)[j]
                    r = np.sqrt(d @ d)
                    q = (mcb if u else mca)[m, a] - (mcb if v else mca)[m, b]
                    dr = r - np.sqrt(q @ q)
                    g = c["mem_weight"][m] * np.exp(-dr * dr / (2 * var))
                    e -= g
                    f[i, u] -= g * dr / var * d / r
                    f[j, v] += g * dr / var * d / r
    return f, e


# memories per window: rows of up to 6 times as many records -- below a piece, about one, two and four pieces, more than
# a block holds
@pytest.mark.parametrize("weighted", [False, True])
@pytest.mark.parametrize("per_window", [1, 5, 6, 11, 21, 22])
@pytest.mark.parametrize("length", [10, 33])
def test_rows(length, per_window, weighted, tmp_path, gpu_lib):
    import torch

    from awsemmd_b200 import engine, synth

    c = synth.chain_arrays(length, 4000 + length + per_window, n_mem_per_window=per_window)
    if weighted:
        c["mem_weight"] = np.linspace(0.5, 1.5, c["n_mem"])
    want_f, want_e = _reference(c)
    ff = synth.forcefield_dir(str(tmp_path / "ff"))
    for prec in ("fp64", "mixed"):
        with engine.AwsemBatch.from_arrays(ff, [c], precision=prec) as s:
            x = torch.tensor(np.ascontiguousarray(c["x"][:, [0, 2, 1]]), device="cuda")
            f, e = torch.empty_like(x), torch.empty(1, dtype=torch.float64, device="cuda")
            fn = s.lib.awsem_fragmem_noalloc
            fn.argtypes = [C.c_void_p] * 5
            assert fn(s.h, x.data_ptr(), f.data_ptr(), e.data_ptr(), torch.cuda.current_stream().cuda_stream) == 0
            torch.cuda.synchronize()
            f = f.cpu().numpy()[:, [0, 2, 1]]
            # an atom gets at most 24 contributions, each rounded to 2^-32; the sums themselves are good to a few
            # hundred units in the last place of the form's type
            eps = 1e-13 if prec == "fp64" else 1e-4
            assert np.abs(f - want_f).max() <= 24 * 2.0 ** -33 + eps * np.abs(want_f).max()
            assert abs(e.item() - want_e) <= 6 * length * 2.0 ** -33 + (1e-13 if prec == "fp64" else 1e-5) * abs(want_e)
            # the engine's own kernel, a block, a warp or a chunk of separations a unit: the same bits
            x0 = c["x"].reshape(-1, 3)
            got = []
            for shapes in ((6, 148, 148, 0), (6, 148, 148, 2), (1, 148, 148, 0), (3, 148, 148, 3)):
                s.set_launch_shapes(shapes)
                got.append(s.compute(x0))
            for g in got[1:]:
                assert np.array_equal(g[0], got[0][0])
                assert abs(g[1][12] - got[0][1][12]) <= 6 * length * 2.0 ** -32
            assert abs(got[0][1][12] - want_e) <= 6 * length * 2.0 ** -33 + (1e-13 if prec == "fp64" else 1e-5) * abs(want_e)
