"""An ensemble whose model fails: nothing is left running on its memory."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def test_a_failed_run_leaves_no_work_in_flight(cuda_device, monkeypatch):
    """The models' memory goes back to the stream the next run builds on, so
    work on any other stream (a batched solve's) must be over by then."""
    from transportse_b200 import ensemble, workloads
    side = torch.cuda.Stream(device=cuda_device)
    ended = torch.cuda.Event()

    def fails(sim, steps, keep, gate, joined=False):
        with torch.cuda.stream(side):
            for _ in range(20):
                torch.cuda._sleep(20_000_000)      # some 10 ms each
                sim.S["P"].mul_(1.0)
            ended.record(side)
        gate.leave()
        raise RuntimeError("stopped by the test")

    monkeypatch.setattr(ensemble, "step_model", fails)
    ens = ensemble.Ensemble([workloads.ensemble_member(seed=3, n_min=16, n_max=20)], device=cuda_device)
    with pytest.raises(RuntimeError, match="stopped by the test"):
        ens.run(1, keep=())
    assert ended.query()
