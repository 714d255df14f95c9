"""Volumes whose rows are shorter than a word, or one to a few voxels longer:
the leaf min/max of the single-volume and the batched pass, run with the
bounds-check build in a child process, loads no word that reaches past the
volume and gives the oracle's block min/max bit for bit.  Slices of one row and
of a whole number of block rows and two, where the last row but one lies in
another block row than the last, at base addresses off the word."""
import os
import subprocess
import sys

import numpy as np
import pytest
import torch

HERE = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(HERE)


@pytest.mark.gpu
def test_short_rows_stay_in_the_volume():
    lib = os.path.join(ROOT, "meshtrex_b200", "libmeshtrex_b200_check.so")
    assert os.path.exists(lib), "build it with `make -C meshtrex_b200/csrc check`"
    r = subprocess.run([sys.executable, os.path.abspath(__file__)], capture_output=True, text=True,
                       env=dict(os.environ, MESHTREX_B200_LIB=lib), timeout=600)
    assert r.returncode == 0, r.stdout[-3000:] + r.stderr[-3000:]
    assert "all rows in the volume" in r.stdout


def main():
    sys.path.insert(0, ROOT)
    sys.path.insert(0, HERE)
    from helpers import TORCH, u32
    from meshtrex_b200 import api
    from oracle import oracle as O
    ctx = api.Context(0)
    rng = np.random.default_rng(3)
    for dtype, widths in ((np.uint8, (1, 2, 3, 4, 5, 6, 7, 9)), (np.uint16, (1, 2, 3, 4))):
        top = np.iinfo(dtype).max
        for X in widths:
            vols, blocks, arrays = [], [], []
            for B, Y, Z in ((2, 1, 4), (2, 4, 2), (2, 6, 3), (3, 5, 4), (8, 10, 9), (16, 18, 3)):
                for offset in range(4 // np.dtype(dtype).itemsize):
                    a = rng.integers(0, top, (Z, Y, X), endpoint=True).astype(dtype)
                    raw = a.reshape(-1).view(np.int16) if dtype == np.uint16 else a.reshape(-1)
                    buf = torch.zeros(a.size + offset, dtype=torch.from_numpy(raw).dtype, device="cuda")
                    buf[offset:] = torch.from_numpy(raw).cuda()
                    vol = buf.view(TORCH[np.dtype(dtype)])[offset:].view(a.shape)
                    mm = api.compute_min_max_mip(ctx, api.wrap_volume(vol), api.push_constants((X, Y, Z), B, 1.0))
                    ctx.synchronize()
                    np.testing.assert_array_equal(
                        u32(mm.all_levels()), O.pyramid(O.minmax_halo(a, B), O.block_grid(a.shape, B)), str((X, Y, Z, B)))
                    mm.free()
                    vols.append(vol)
                    blocks.append(B)
                    arrays.append(a)
            # the batch: its active blocks follow from the same min/max
            iso = float(top // 2)
            b = api.Batch(ctx, vols, blocks, [(v, iso) for v in range(len(vols))], use_graph=False)
            b.run()
            jobs, _ = b.results()
            for a, B, j in zip(arrays, blocks, jobs):
                assert j["meshletCount"] == len(O.extract(a, B, iso).ids), (a.shape, B)
            b.close()
            ctx.synchronize()
    ctx.close()
    print("all rows in the volume", flush=True)


if __name__ == "__main__":
    main()
