"""The exact sweep's recombination of the eight order accumulators, replayed on
the CPU with the word sizes the kernel uses, and its conversion's scaling on
the GPU."""
import numpy as np
import pytest

M32, M64 = 2 ** 32 - 1, 2 ** 64 - 1
BIAS = 0x43400000                                # FP32 bits of 1.5 * 2^23 units of 2^-16
PAIR = (257 * BIAS) & M32


def constants(esum):
    """tc_filter_digits' k64 and k67 from the sums of the filter's digits e_0 .. e_7."""
    c = [128 * sum(esum[:k + 1]) for k in range(8)]
    k64 = PAIR * (2 ** 38 + 2 ** 22 + 2 ** 6) + sum(c[k] << (46 - 8 * k) for k in range(6))
    return (-k64) & M64, (512 - PAIR - (256 * c[6] + c[7])) & M32


def recombine(acc, k64, k67):
    """horner_bal: neighbouring orders in one 32-bit word, joined modulo 2^64."""
    b = [(BIAS + int(v)) & M32 for v in acc]
    w01, w23, w45 = ((256 * b[k] + b[k + 1]) & M32 for k in (0, 2, 4))
    lo = (256 * b[6] + b[7] + k67) & M32
    lo = (lo - 2 ** 32 if lo >> 31 else lo) >> 10
    v = (k64 + w45 * 64 + w23 * 2 ** 22 + lo + (((w01 * 64) & M32) << 32)) & M64
    return v - 2 ** 64 if v >> 63 else v


@pytest.mark.parametrize('taps', [16, 29, 32])
def test_recombination_of_offset_digits(taps):
    """Data digits enter the accumulators as bytes d + 128: the recombination gives the sum over
    the balanced digits, exactly, and zero for zero data."""
    r = np.random.default_rng(taps)
    for i in range(60):
        e = r.integers(-128, 128, (8, taps)) >> int(r.integers(0, 3))
        d = r.integers(-128, 128, (8, taps)) if i else np.zeros((8, taps), dtype=int)
        d[0] >>= 1                                # |X| < 2^62
        e[0] >>= 1
        acc = [sum(int((e[t] * (d[k - t] + 128)).sum()) for t in range(k + 1)) for k in range(8)]
        true = [sum(int((e[t] * d[k - t]).sum()) for t in range(k + 1)) for k in range(8)]
        pos = 255 * max(int(np.where(e > 0, e, 0).sum()), int(np.where(e < 0, -e, 0).sum()))
        if pos > 2 ** 22:                        # tc_filter_digits cuts such digits again
            continue
        assert max(abs(v) for v in acc) <= 2 ** 22
        Y = sum(true[k] * 2 ** (46 - 8 * k) for k in range(6)) + ((true[6] * 256 + true[7] + 512) >> 10)
        if abs(Y) >= 2 ** 63:                    # the filter scale keeps |Y| below 2^62
            continue
        assert recombine(acc, *constants([int(v.sum()) for v in e])) == Y
        assert i or Y == 0


@pytest.mark.parametrize('acc', [[2 ** 22] * 8, [-2 ** 22] * 8, [0] * 8, [2 ** 22, -2 ** 22] * 4])
def test_recombination_at_the_accumulators_limits(acc):
    Y = sum(acc[k] * 2 ** (46 - 8 * k) for k in range(6)) + ((acc[6] * 256 + acc[7] + 512) >> 10)
    assert (recombine(acc, *constants([0] * 8)) - Y) % 2 ** 64 == 0


def test_a_byte_is_an_exact_subnormal():
    """FP16 bits 0x00uu are u 2^-24; digits times 2^8 and the bias 3 * 8 * 8 share the unit 2^-16."""
    u = np.arange(256, dtype=np.uint16).view(np.float16).astype(float)
    assert np.array_equal(u, np.arange(256) * 2.0 ** -24)
    assert np.array_equal(np.float16(256.0 * np.arange(-128, 128)).astype(float), 256.0 * np.arange(-128, 128))
    assert int(np.array(192.0, dtype=np.float32).view(np.uint32)) == BIAS
    assert 3 * float(np.uint16(0x4800).view(np.float16)) ** 2 == 192.0 == 1.5 * 2 ** 23 * 2.0 ** -16


@pytest.mark.gpu
@pytest.mark.parametrize('k', [-1010, -960, -900, 0, 900, 955, 1000])
@pytest.mark.parametrize('op', ['d_s0s0_1d_sym8_md', 'd_kin'])
def test_power_of_two_scaling_is_exact(pkg, op, k):
    """Exact sweeps scale with their lines: x 2^k gives y 2^k bit for bit, on both sides of the
    scales where the kernel changes its conversion (2^se with se in [-1022, 961]); a line of
    zeros stays zero.  The inputs are multiples of 2^-20 in [-1, 1) and every result is normal."""
    from boast_lig_gb300 import inputs
    n = [33, 20, 24]
    x = np.floor(inputs.uniform(9, int(np.prod(n))) * 2 ** 20) * 2.0 ** -20
    x.reshape(n[::-1])[3, 5] = 0.0

    def run(v):
        y, w1, w2 = np.zeros_like(v), np.zeros_like(v), np.zeros_like(v)
        with pkg.mode(pkg.MODE_TC_EXACT):
            if op == 'd_kin':
                pkg.Kernel(op).run(3, n, [0, 0, 0], v, y, w1, w2, [0.5, 0.25, 1.0], 0.0, 0.0)
            else:
                pkg.Kernel(op).run(3, 0, n, 0, n, n, 1, v, y, 1.0, 0.0, 0.0)
        return y

    y0, yk = run(x), run(np.ldexp(x, k))
    big = np.abs(np.ldexp(y0, k)) >= 2.0 ** -1021
    assert big.mean() > 0.9
    assert np.array_equal(yk[big], np.ldexp(y0, k)[big])
    if op != 'd_kin':
        assert not yk.reshape(n[::-1])[3, 5].any()
