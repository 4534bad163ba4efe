"""bench.py's rooflines: a rate only from bytes that were recorded for the template
count at hand, and never from the bytes of updates that the rounds do not make."""
from types import SimpleNamespace

import pytest


def _bench():
    return pytest.importorskip('bench')


def test_no_rate_without_recorded_traffic(monkeypatch):
    bench = _bench()
    monkeypatch.setattr(bench, 'profile_traffic', lambda name: None)
    setup = SimpleNamespace(C=384, K=6, nt=61, NT=60000)
    _, mp_bytes = bench.algorithmic_work(setup, 9300.0, 400)
    r = bench.rounds_roofline(400, 0.70, mp_bytes, 6542.4, 'measured')
    assert r['achieved'] is None and r['frac'] is None and r['traffic'] is None and r['traffic_source'] is None
    p = bench.path_roofline(setup, 9300.0, 400, 1040.0, 6542.4, 1681.1, 'measured', bench.rounds_traffic(400))
    assert p['bytes_per_rec_s'] is None and p['gbs'] is None and p['frac_hbm'] is None
    assert p['bound'] == 'tensor' and p['frac'] == p['frac_tensor'] > 0


def test_rate_of_the_recorded_traffic(monkeypatch):
    bench = _bench()
    asked = []
    monkeypatch.setattr(bench, 'profile_traffic', lambda name: asked.append(name) or 1_800_000_000)
    r = bench.rounds_roofline(800, 2.0, 23.4e9, 6542.4, 'measured')
    assert asked == ['k_mp_lazy_384ch_800t.md']
    assert r['achieved'] == pytest.approx(900.0) and r['frac'] == pytest.approx(900.0 / 6542.4)
    setup = SimpleNamespace(C=384, K=6, nt=61, NT=60000)
    p = bench.path_roofline(setup, 19700.0, 800, 540.0, 6542.4, 1681.1, 'measured', 1_800_000_000)
    # half a batch per recording-second: int16 rows, the scores written, half of the rounds' bytes
    assert p['bytes_per_rec_s'] == pytest.approx(2 * 384 * 30000 + 4 * 800 * 30000 + 0.9e9)
    assert p['frac_hbm'] == pytest.approx(p['bytes_per_rec_s'] * 540.0 / 1e9 / 6542.4) and p['frac_hbm'] < 1
