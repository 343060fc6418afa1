"""awsem_fragmem_noalloc: a warp a unit, a warp pair a unit and the engine's
own kernel give the same bits, and a handle whose form has not run yet can be
captured once any handle has called."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("weighted", [False, True])
def test_forms_agree_and_capture(weighted, tmp_path, gpu_lib):
    import torch

    from awsemmd_b200 import engine, synth

    ff = synth.forcefield_dir(str(tmp_path / "ff"))
    handles = []
    for prec, per in (("mixed", 20), ("mixed", 1), ("fp64", 20)):  # 120, 6 records a row; a block a row
        c = synth.chain_arrays(77, 60, n_mem_per_window=per)
        if weighted:
            c["mem_weight"] = np.linspace(0.1, 1.5, c["n_mem"])
        handles.append((engine.AwsemBatch.from_arrays(ff, [c], precision=prec), c))
    fn = handles[0][0].lib.awsem_fragmem_noalloc
    fn.argtypes = [C.c_void_p] * 5
    for k, (s, c) in enumerate(handles):
        x0 = c["x"].reshape(-1, 3)
        want = s.compute(x0)[1][12]
        x = torch.tensor(np.ascontiguousarray(c["x"][:, [0, 2, 1]]), device="cuda")
        f, e = torch.empty_like(x), torch.empty(1, dtype=torch.float64, device="cuda")
        stream = torch.cuda.Stream()
        torch.cuda.synchronize()
        if k == 0:
            assert fn(s.h, x.data_ptr(), f.data_ptr(), e.data_ptr(), stream.cuda_stream) == 0
        else:
            g = torch.cuda.CUDAGraph()
            with torch.cuda.graph(g, stream=stream):
                assert fn(s.h, x.data_ptr(), f.data_ptr(), e.data_ptr(), torch.cuda.current_stream().cuda_stream) == 0
            g.replay()
        torch.cuda.synchronize()
        assert abs(e.item() - want) <= 1e-12 * abs(want)  # the same parts; their sum over residues rounds otherwise
        if k == 1:
            s.set_launch_shapes((1, 148, 148, 0))  # six separations a unit: 36 records, a warp pair
            f2, e2 = torch.empty_like(f), torch.empty_like(e)
            assert fn(s.h, x.data_ptr(), f2.data_ptr(), e2.data_ptr(), stream.cuda_stream) == 0
            torch.cuda.synchronize()
            assert torch.equal(f, f2) and torch.equal(e, e2)
    for s, _ in handles:
        s.close()
