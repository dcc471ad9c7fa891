"""The chunk tables a run hands to the device, against the per-step expressions they restate: clock, source values and
DFT phases equal bit for bit."""
import math

import numpy as np
import pytest

from opensol_b200.constants import DTYPE
from opensol_b200.monitors import dft_phase_table, step_clock
from opensol_b200.sources import ContinuousWave, GaussianPulse, LineSource, RickerWavelet, temporal_values


def test_step_clock_accumulates_step_by_step():
    for t, dt, n in ((0.0, 4.7e-17, 1), (3.1e-14, 4.6699e-17, 5000), (1e-13, 1.9e-17, 777)):
        half, full, end = step_clock(t, dt, n)
        x = t
        for k in range(n):
            assert half[k] == x + 0.5 * dt
            x = x + dt
            assert full[k] == x
        assert end == x


@pytest.mark.parametrize('temporal', [GaussianPulse(1.934e14, 0.5), GaussianPulse(5e14, 0.8), ContinuousWave(3e14),
                                      RickerWavelet(2e14)])
def test_source_values_equal_the_scalar_calls(temporal):
    times = step_clock(0.0, 4.67e-17, 20_000)[0]
    values = temporal_values(temporal, times)
    assert values.tolist() == [temporal(float(t)) for t in times]
    source = LineSource('y', 3, temporal, amplitude=0.7)
    got = source.values(times)
    assert got.dtype == DTYPE
    assert got.tolist() == [float(DTYPE(source.amplitude * temporal(float(t)))) for t in times]


@pytest.mark.parametrize('nf', [1, 2, 3, 4, 7, 8, 16])
def test_phase_table_equals_one_sample_at_a_time(nf):
    omega = 2 * np.pi * np.linspace(1.3e14, 5e14, nf)
    times = [k * 27 * 4.67e-17 for k in range(1, 2001)]
    table = dft_phase_table(omega, times, 27 * 4.67e-17)
    for q, t in enumerate(times):
        phase = -omega * float(t)
        np.testing.assert_array_equal(table[q, :, 0], (np.cos(phase) * (27 * 4.67e-17)).astype(np.float32))
        np.testing.assert_array_equal(table[q, :, 1], (np.sin(phase) * (27 * 4.67e-17)).astype(np.float32))
    assert math.isfinite(float(table.sum())) and dft_phase_table(omega, [], 1.0).shape == (0, nf, 2)
