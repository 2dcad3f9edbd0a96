"""Writes trd_kat.npz, the fixture of tests/test_gpu_transform_golden.py, with a given build of the
library on a GPU:

    python tests/golden/make_trd_golden.py LIBRARY [OUTPUT]

The fixture holds the outputs of the library built from commit 1a106a5 (`git archive 1a106a5`, then
`python -m libvc1_b200.build` there), the last one whose transform RD, DQUANT search and intra
reconstruction ran one parent block per thread; those had been compared with the reference's own
functions bit for bit (test_gpu_transform_rd.py, test_gpu_dquant.py and test_gpu_intra.py, where
oracle/_ref is built). Without OUTPUT nothing is written: the build's outputs are compared with the
fixture, every array by its bytes.
"""
import os
import sys

import numpy as np

HERE = os.path.dirname(os.path.abspath(__file__))
sys.path[:0] = [os.path.dirname(os.path.dirname(HERE)), os.path.dirname(HERE)]

import test_gpu_transform_golden as golden  # noqa: E402
from libvc1_b200.api import CudaComputeContext  # noqa: E402


def main(library, output=None):
    ctx, err = CudaComputeContext.create(0, library=library)
    if ctx is None:
        raise SystemExit(err)
    arrays = {f"c{i}.{k}": v for i in range(len(golden.CASES)) for k, v in golden.results(ctx, i).items()}
    ctx.close()
    if output:
        np.savez_compressed(output, **arrays)
        return 0
    want = np.load(golden.GOLDEN)
    bad = [k for k in sorted(set(want.files) | set(arrays))
           if k not in arrays or k not in want.files or arrays[k].dtype != want[k].dtype or
           arrays[k].tobytes() != want[k].tobytes()]
    print("differs: " + ", ".join(bad) if bad else f"{len(arrays)} arrays equal the fixture")
    return 1 if bad else 0


if __name__ == "__main__":
    sys.exit(main(*sys.argv[1:]))
