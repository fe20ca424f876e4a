"""The chemical-potential search (csrc/mu.cu) when its blocks give up a wait, as they do
where another thread's kernel holds some SMs for seconds: it starts again from the same
state, with the result of an undisturbed search.  The first wait is made one cycle long
(PYRPA_GB_MU_WAIT), which no search on several blocks gets by with."""
import numpy as np
import pytest

from test_gpu_even import F, model, step_args  # noqa: F401


@pytest.mark.gpu
@pytest.mark.parametrize("dims", [(1, 32, 32, 1, 300), (2, 16, 16, 1, 64), (5, 8, 8, 1, 64)])
def test_search_starts_again_after_a_wait_given_up(F, monkeypatch, dims):  # noqa: F811
    m = model(*dims)

    def run():
        n = F.kernel_launches()
        sg, mu = F.mkself(*step_args(m), scf_loop=2, eps=0.0, pp=0.5, sw_rescale=True)
        return sg, mu, F.kernel_launches() - n

    run()  # tables and plans of the first call
    sg, mu, n = run()
    monkeypatch.setenv("PYRPA_GB_MU_WAIT", "1")
    wsg, wmu, wn = run()
    assert wn > n
    assert wmu == mu
    assert np.array_equal(wsg, sg)
