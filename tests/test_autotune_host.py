"""The autotuner's choice, with the timing replaced: the default tiles are
among what it times, and no combination is timed twice where a setting does
not act."""
import pytest

from lcode3d_b200 import batch as B


@pytest.mark.parametrize('precision', ['fp64', 'fft32'])
def test_autotune_can_keep_the_default(monkeypatch, precision):
    timed = []

    def fake(spec, prec, form, tiles, steps):
        timed.append((form, *tiles))
        assert prec == precision
        if form == 'dense' and precision == 'fft32':
            return None
        # the default height is fastest; the FFT setting acts in float32 passes only
        return 1.0 + tiles[0] / 10 + (form == 'dense') + (tiles[1] / 100 if precision == 'fft32' else 0)
    monkeypatch.setattr(B, '_time_sim', fake)
    choice, timings = B.autotune([161], precision=precision)
    assert choice[161] == {'transform': 'fft', 'deposit_rows': 0, 'fft_ctas_per_sm': 0}
    assert len(timed) == len(set(timed))
    ctas = {t[2] for t in timed if t[0] == 'fft'}
    assert ctas == (set(B.TILE_CHOICES['fft_ctas_per_sm']) if precision == 'fft32' else {0})
    for rows in B.TILE_CHOICES['deposit_rows']:
        for per_sm in B.TILE_CHOICES['fft_ctas_per_sm']:
            assert timings[161][f'fft rows={rows} fft_per_sm={per_sm}'] >= 1.0
