"""Device memory of a batch's scratch: mixed-event rows have no fixed-point
columns (64 bytes of a row)."""
import pytest

from hadronic_afterburner_toolkit_gb300 import engine

pytestmark = pytest.mark.gpu


def test_bytes_of_a_mixed_row():
    torch = pytest.importorskip("torch")
    n = 4_000_000
    gen = torch.Generator(device="cuda").manual_seed(1)
    p = torch.randn(3, n, generator=gen, device="cuda", dtype=torch.float64) * 0.3
    a = [*p, torch.sqrt(0.02 + (p * p).sum(0))]
    b = [c[:64].contiguous() for c in a]
    eng = engine.Engine()
    eng.bin_mixed(b, b, device=True)  # what every context has
    eng.sync()
    before = torch.cuda.mem_get_info()[0]
    eng.bin_mixed(a, b, device=True)
    eng.sync()
    used = before - torch.cuda.mem_get_info()[0]
    # table 64, terms 24, order 4, sort keys 16, positions 8, and as much again
    # as keys and positions for the sort; an eighth over for the growth
    assert used <= 1.125 * n * (64 + 24 + 4 + 2 * (16 + 8))
    assert eng.hist()["den"].sum() > 1e5
    eng.close()
