"""The V-cycle's coarsest sweeps divide by 3 as q = t i, q + (t - 3 q) i with i = fl(1/3) and fused multiply-adds
(dividirViz, pcg.cu): for every significand of t that is t / 3 correctly rounded.  Whole numbers, in quarters and in
2^-27, stand for the floats; the quotients of t in [2^23, 2^24) have their last place at 1/4 or 1/2."""
import numpy as np

TERCO = 11184811  # fl(1/3) 2^25


def arredondar(v, bits):
    """v 2^-bits rounded to the nearest whole number, ties to even."""
    metade = np.int64(1) << (bits - 1)
    q, resto = v >> bits, v & (2 * metade - 1)
    return q + ((resto > metade) | ((resto == metade) & ((q & 1) == 1)))


def test_todos_os_significandos():
    assert np.float32(TERCO) * np.float32(2.0**-25) == np.float32(1) / np.float32(3)
    t = np.arange(1 << 23, 1 << 24, dtype=np.int64)
    p = t * TERCO
    q = np.where(p < 1 << 47, arredondar(p, 23), 2 * arredondar(p, 24))  # t i, in quarters
    resto = 4 * t - 3 * q
    assert np.abs(resto).max() < 1 << 24  # exact in a float
    s = (q << 25) + resto * TERCO  # q + (t - 3 q) i, in 2^-27
    r = np.where(s < 1 << 49, arredondar(s, 25), 2 * arredondar(s, 26))
    # t / 3 to the nearest: no quotient lies half-way between two floats
    certo = np.where(t < 3 << 22, (8 * t + 3) // 6, 2 * ((4 * t + 3) // 6))
    assert np.array_equal(r, certo)
