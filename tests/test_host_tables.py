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


class _Numpy:
    """A waveform whose values are numpy float64 (its product with a numpy float32 is taken in float64)."""

    def __call__(self, t):
        return np.sin(np.float64(3e14) * t) * np.float64(0.3)


@pytest.mark.parametrize('n', [0, 1, 2, 15, 16, 17, 300])
@pytest.mark.parametrize('temporal, amplitude', [
    (_Numpy(), None), (GaussianPulse(2e14, 0.5), 0.7), (GaussianPulse(2e14, 0.5), np.float64(0.7)),
    (GaussianPulse(np.float32(2e14), 0.5), None), (ContinuousWave(np.float32(3e14)), None), (RickerWavelet(2e14), 2)])
def test_any_waveform_amplitude_and_length(temporal, amplitude, n):
    """Lengths around the line between the two ways, waveforms of the caller's own, amplitudes set later."""
    source = LineSource('y', 3, temporal, amplitude=0.7)
    if amplitude is not None:
        source.amplitude = amplitude
    half, full, end = step_clock(2e-15, 4.67e-17, n)
    x = 2e-15
    for k in range(n):
        assert half[k] == x + 0.5 * 4.67e-17
        x = x + 4.67e-17
        assert full[k] == x
    assert end == x and half.shape == full.shape == (n,)
    got = source.values(half)
    assert got.dtype == DTYPE and got.shape == (n,)
    assert got.tolist() == [float(DTYPE(source.amplitude * temporal(float(t)))) for t in half]


def test_short_chunks_take_no_array_detour():
    """A chunk of one step is as cheap as the loop it restates: no phase arithmetic without samples, no native call."""
    def refuse(*_):
        raise AssertionError('a chunk of one step went through the arrays')
    pulse = GaussianPulse(2e14, 0.5)
    pulse.at = refuse
    LineSource('y', 3, pulse).values(step_clock(0.0, 4.67e-17, 1)[0])

    class Omega:
        size = 4

        def __neg__(self):
            refuse()
        __getitem__ = __mul__ = __rmul__ = refuse
    assert dft_phase_table(Omega(), [], 1.0).shape == (0, 4, 2)
