"""The library's launch counter: a step that is launched kernel by kernel counts as many
as the kernel nodes of its replayed graph."""
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


@pytest.mark.parametrize("method,rule,n", [("fp64", "", 300), ("fp64", "", 3000),
                                           ("mixed", "", 1000), ("mixed", "", 5000),
                                           ("bh", "", 3000), ("bh", "ref", 3000),
                                           ("bh", "quad", 40_000), ("bh", "", 600_000)])
def test_direct_steps_count_what_replays_count(nb, method, rule, n):
    cfg = nb.Config(method={"fp64": nb.DIRECT_FP64, "mixed": nb.DIRECT_MIXED,
                            "bh": nb.BARNES_HUT}[method], G=1.0, softening=0.01, theta=0.6,
                    flags={"": 0, "ref": nb.BH_REFERENCE_OPENING, "quad": nb.BH_QUADRUPOLE}[rule])
    state = nb.plummer(n, seed=n)
    side = torch.cuda.Stream()
    counts = []
    for stream in (None, side.cuda_stream):  # the legacy default stream is not captured
        with nb.Sim(cfg, capacity=n, stream=stream) as s:
            s.load(*state)
            s.step(nb.LEAPFROG, 1e-3, 4)
            before = nb.kernel_launch_count()
            s.step(nb.LEAPFROG, 1e-3, 1)
            counts.append(nb.kernel_launch_count() - before)
    assert counts[0] == counts[1] > 0
