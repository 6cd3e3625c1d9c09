"""A batch counts the kernels that a replay launches, in its statistics and in
the library's counter."""
import pytest

from test_gpu_table_forms import job, plan

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("Ls", [(10,), (10, 6, 13)])
def test_batch_counts_its_launches(gpu, Ls):
    """A plan's run launches 2 kernels for the per-z tables, 2 rotations, one
    translation for each four columns, the poses and the fit; a batch puts the
    rotations of one gamma group and the fits in one launch each."""
    js = [job(gpu, L, 12, 60, L) for L in Ls]
    plans = [plan(gpu, j, precision=1) for j in js]
    b = gpu.Batch(plans)
    groups = len({gpu.load().sxsk_rotate_group(L, gpu.tiles_default(L, 12)[1]) for L in Ls})
    want = groups + sum(2 + (L + 4) // 4 + 1 for L in Ls) + 1
    before = gpu.launch_count()
    b.run()
    b.run()
    assert b.stats()["launches"] == want
    assert gpu.launch_count() - before == 2 * want
    b.close()
    for p in plans:
        p.close()
