"""A window's result does not depend on the other windows of its batch: alone,
beside small ones, and beside one with a camera whose blocks do not fit in
shared memory (about 1,350 of them do), for which the Schur rows take another
form."""

import numpy as np
import pytest

from g2o_b200 import synth


# rows with up to 4, up to 8 and more off-diagonal blocks; cameras with fewer
# and with more blocks than a CTA of the other form has threads (512)
@pytest.mark.gpu
@pytest.mark.parametrize("cams,points", [(2, 40), (4, 700), (6, 300), (9, 1200), (10, 150), (14, 900)])
def test_same_bits_alone_and_beside_a_large_camera(cams, points):
    from g2o_b200 import backend
    w = synth.bundle_adjustment(cams, points, seed=cams)
    other = synth.bundle_adjustment(5, 80, seed=50)
    large = synth.bundle_adjustment(3, 2500, seed=51)

    def run(batch):
        c = backend.CudaWindows(batch)
        c.optimize(4)
        e = c.estimates_all()[0]
        c.close()
        return e

    alone = run([w])
    for batch in ([w, other], [w, large], [w, other, large]):
        assert all(np.array_equal(a, b) for a, b in zip(alone, run(batch)))
