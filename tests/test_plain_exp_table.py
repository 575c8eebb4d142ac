"""The table of k_plain_step's exponential (csrc/bx_plain.cuh), read from the
source: 2^(j/64) rounded to nearest, the rest relative to it, and ln2 / 64 in
two parts whose first times a 17-bit integer is exact."""
import pathlib
import re
from decimal import Decimal, getcontext
from fractions import Fraction

SRC = pathlib.Path(__file__).resolve().parent.parent / 'betse_gb300' / 'csrc' / 'bx_plain.cuh'
HEX = r'(-?0x[0-9a-f.]+p[-+]\d+)'


def test_table_and_constants():
    getcontext().prec = 60
    text = SRC.read_text()
    tab = re.findall(r'\{%s, %s\}' % (HEX, HEX), text[text.index('kExpTab[64]'):text.index('struct PlainExp ')])
    assert len(tab) == 64
    ln2 = Decimal(2).ln()
    for j, (hi, rel) in enumerate(tab):
        v = (ln2 * j / 64).exp()
        h = float.fromhex(hi)
        assert h == float(v), j
        r = (v - Decimal(h)) / Decimal(h)
        assert abs(Decimal(float.fromhex(rel)) - r) < Decimal(2) ** -105, j
    hi, lo = (float.fromhex(x) for x in re.search(r'kLn2Hi = %s, kLn2Lo = %s' % (HEX, HEX), text).groups())
    inv = float.fromhex(re.search(r'kInvLn2 = %s' % HEX, text).group(1))
    assert abs(Decimal(hi) + Decimal(lo) - ln2 / 64) < Decimal(2) ** -97
    assert inv == float(64 / ln2)
    for n in (1, 3, 2 ** 16 - 1, 2 ** 17 - 1):
        assert Fraction(n * hi) == n * Fraction(hi)
