"""The amplitude kernels' paths beyond the ordinary phase-passed seed: sides under the listing floor (a second pass
without it), thresholds on and next to an amplitude, thresholds that drop or keep every seed.  Oracle values, exactly."""
import numpy as np
import pytest

import libs

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def any_phase(dsg):
    """96 seeds at any y-phase, their oracle amplitudes: maxima both under and over the floor of 0.24."""
    seeds = np.array([libs.mix(77 * 10**12 + k) for k in range(96)], dtype=np.uint64)
    return seeds, *libs.orc_gate(seeds, True, *dsg.gate_taps())


def test_amps_of_any_phase(dsg, any_phase):
    seeds, opre, ofull = any_phase
    pre, full = dsg.gate_amps(seeds)
    assert np.array_equal(pre, opre) and np.array_equal(full, ofull)
    assert (opre < 0.24).any() and (opre > 0.24).any()


@pytest.mark.parametrize("n", [1, 2, 95])
def test_amps_of_few_seeds(dsg, any_phase, n):
    seeds, opre, ofull = any_phase
    pre, full = dsg.gate_amps(seeds[-n:])
    assert np.array_equal(pre, opre[-n:]) and np.array_equal(full, ofull[-n:])


def test_thresholds_on_an_amplitude(dsg):
    """A gate whose thresholds equal one seed's amplitudes passes it; one float above either, it does not."""
    start, count = 10**12, 1 << 15
    seeds = np.array([libs.mix(start + k) for k in range(count)], dtype=np.uint64)
    ph, _ = libs.orc().phase(seeds)
    s = seeds[ph <= np.float64(np.float32(0.06))]
    pre, full = libs.orc_gate(s, True, *dsg.gate_taps())
    p, f = pre[:, 0] + pre[:, 1], full[:, 0] + full[:, 1]
    for i in np.argsort(p)[[5, len(p) // 2, -5]]:
        for pthr, amp in [(p[i], f[i]), (np.nextafter(p[i], np.float32(9)), f[i]), (p[i], np.nextafter(f[i], np.float32(9)))]:
            got, a, counts, rc = dsg.gate_run(start, count, pthr=float(pthr), amp=float(amp))
            want = (p >= pthr) & (f >= amp)
            assert rc == 0 and np.array_equal(got, np.sort(s[want])) and np.array_equal(a, f[want][np.argsort(s[want])])
            assert int(counts[2]) == int((p >= pthr).sum())


@pytest.mark.parametrize("pthr,amp", [(-1.0, -1.0), (0.0, 0.5), (0.3, 9.0), (9.0, 0.0)])
def test_thresholds_that_keep_or_drop_all(dsg, pthr, amp):
    start, count = 3 * 10**12, 3000
    seeds = np.array([libs.mix(start + k) for k in range(count)], dtype=np.uint64)
    ph, _ = libs.orc().phase(seeds)
    s = seeds[ph <= np.float64(np.float32(0.06))]
    pre, full = libs.orc_gate(s, True, *dsg.gate_taps())
    p, f = pre[:, 0] + pre[:, 1], full[:, 0] + full[:, 1]
    got, a, counts, rc = dsg.gate_run(start, count, pthr=pthr, amp=amp)
    assert rc == 0 and [int(c) for c in counts[1:]] == [len(s), int((p >= np.float32(pthr)).sum()), int(((p >= np.float32(pthr)) & (f >= np.float32(amp))).sum())]
    want = (p >= np.float32(pthr)) & (f >= np.float32(amp))
    assert np.array_equal(got, np.sort(s[want]))
