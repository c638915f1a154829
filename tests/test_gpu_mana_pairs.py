"""Mana of pure states: two X-strings, a multiple of a row (3^ceil(L / 2) elements) apart, share a
transform.  Ranges longer than that distance, off its multiples, hold X-strings with and
without a partner: their sum is that of ranges of one X-string, which have none."""
import pytest

from conftest import rand_state

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("L,begin,length", [(5, 50, 150), (6, 20, 65), (6, 598, 131), (7, 50, 200), (7, 2056, 131),
                                            (8, 50, 200), (8, 6430, 131), (8, 3000, 82), (9, 100, 400)])
def test_ranges_with_partners_equal_single_x_strings(ctx, L, begin, length):
    row = 3 ** ((L + 1) // 2)
    distance = (length + 2 * row - 1) // (2 * row) * row
    assert distance < length and begin + length <= 3 ** L  # some X-strings have a partner
    psi = rand_state(3 ** L, 980 + L)
    singles = sum(ctx.mana_pure_range(psi, x, x + 1).sum() for x in range(begin, begin + length))
    assert ctx.mana_pure_range(psi, begin, begin + length).sum() == pytest.approx(singles, rel=1e-13)
