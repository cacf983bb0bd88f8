"""Which form of the full sum 'auto' takes, against both forms' measured times (B200, us)."""
import pytest

from hotspice_b200.core import fft_is_faster


# cells, magnets, window, slots, minimum image, direct sum, convolution
@pytest.mark.parametrize('cells,magnets,window,slots,wrap,direct,fft', [
    (576, 576, 576, 1, False, 100.8, 27.5),            # square 24 x 24, uncut
    (4096, 4096, 121, 1, True, 34.9, 26.8),            # square 64 x 64
    (4096, 4096, 225, 1, False, 43.0, 25.7),
    (40000, 40000, 121, 1, False, 28.7, 39.6),         # square 200 x 200
    (40000, 40000, 169, 1, True, 51.1, 39.5),
    (40000, 40000, 625, 1, False, 121.3, 39.3),
    (65536, 65536, 169, 1, False, 38.8, 40.2),         # square 256 x 256
    (250000, 250000, 121, 1, False, 61.2, 44.7),       # square 500 x 500
    (1000000, 1000000, 225, 1, False, 360.9, 115.6),   # square 1000 x 1000
    (40000, 20000, 169, 2, False, 34.3, 44.5),         # pinwheel 200 x 200
    (40000, 20000, 169, 2, True, 47.3, 43.7),
    (1000000, 500000, 169, 2, False, 231.9, 138.2),    # pinwheel 1000 x 1000
    (240, 91, 117, 6, False, 28.3, 41.6),              # kagome 16 x 15
    (992, 377, 992, 6, False, 180.5, 47.6),            # kagome 32 x 31, uncut
    (65280, 24806, 117, 6, False, 26.6, 67.3),         # kagome 256 x 255
    (489300, 185934, 153, 6, False, 99.7, 127.9),      # kagome 700 x 699
    (999000, 379620, 231, 6, False, 301.4, 216.9),     # kagome 1000 x 999
    (16384, 16384, 121, 4, False, 30.4, 48.8),         # open square 128 x 128
    (256, 256, 256, 4, False, 82.2, 37.4),             # open square 16 x 16, uncut
])
def test_rule_takes_the_faster_form(cells, magnets, window, slots, wrap, direct, fft):
    taken = fft if fft_is_faster(cells, magnets, window, slots, wrap) else direct
    assert taken <= 1.1 * min(direct, fft)


def test_many_sublattices_of_a_small_lattice_stay_with_the_direct_sum():
    # 128 slots: the convolution transforms each of them
    assert not fft_is_faster(1024, 1024, 1024, 128, False)
    assert fft_is_faster(96 * 96, 96 * 96, 96 * 96, 128, False)
