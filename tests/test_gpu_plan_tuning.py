"""A plan's knobs: the automatic grab can be asked for, and a knob that is not
named keeps the plan's own default."""
import pytest

from bcl_b200 import autotune, gen
from oracle import oracle as O

from gpu_util import assert_csr_identical

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def cuda():
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")


@pytest.mark.parametrize("tuning,want", [({"light_ub": 256}, (0, 4, 14)), ({"long_seg": 6}, (0, 4, 6)),
                                         ({"grab": 2}, (2, 4, 14)), ((0, 3, 28), (0, 3, 28))])
def test_unnamed_knobs_keep_their_defaults(monkeypatch, tuning, want):
    from bcl_b200.containers import BlockCustom, SpgemmPlan, SPMatrix, spgemm
    assert autotune.DEFAULT == (0, 4, 14) and 0 in autotune.CANDIDATES["grab"]
    seen, tune = [], SpgemmPlan.tune
    monkeypatch.setattr(SpgemmPlan, "tune", lambda self, *a: (seen.append(a), tune(self, *a)))
    a = gen.rmat(10, seed=3)
    A = SPMatrix.from_csr(a, BlockCustom((512, 512)))
    assert_csr_identical(spgemm(A, A, tuning=tuning).get(), *O.gemm_tiled(a, a, 512, 512, 512))
    assert seen == [want]


@pytest.mark.parametrize("grab", [-1, 65])
def test_grab_out_of_range(grab):
    from bcl_b200._lib import BclxError
    from bcl_b200.containers import BlockCustom, SPMatrix, spgemm_symbolic
    A = SPMatrix.from_csr(gen.erdos_renyi(64, 3, seed=1), BlockCustom((64, 64)))
    plan = spgemm_symbolic(A, A)[0]
    with pytest.raises(BclxError):
        plan.tune(grab, 4, 14)
    plan.close()
