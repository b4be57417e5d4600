"""CPU: the ranges that the 32-bit indices of the det <-> CSF transforms rely on
(pyscf-forge_b200/csrc/transform_tile.cuh): in every space of at most 2^32
determinants (the limit of the determinant addressing) each npair block's spin
function table, mask offsets and CSF offsets stay below 2^32.  The table does
pass 2^31, so its index has to be unsigned."""
import os
import re
from math import comb

from conftest import ROOT


def _blocks(norb, na, nb):
    for npair in range(max(0, na + nb - norb), min(na, nb) + 1):
        nspin = na + nb - 2 * npair
        if nspin > 32:  # refused by the spin function table
            continue
        nconf = comb(norb, npair) * comb(norb - npair, nspin)
        yield nspin, nconf, comb(nspin, na - npair)


def test_block_tables_fit_32_bits():
    most = 0
    for norb in range(1, 64):
        for na in range(norb + 1):
            for nb in range(na + 1):
                if comb(norb, na) * comb(norb, nb) > 2 ** 32:
                    continue
                for nspin, nconf, ndet in _blocks(norb, na, nb):
                    two_s = range(na - nb, nspin + 1, 2)
                    ncsf = max((comb(nspin, (nspin - s) // 2) - comb(nspin, (nspin - s) // 2 - 1)
                                if s < nspin else 1) for s in two_s)
                    assert ncsf <= ndet and nconf * ndet <= 2 ** 32
                    most = max(most, ndet * ncsf)
    assert 2 ** 31 < most < 2 ** 32


def test_table_index_is_unsigned():
    """Both products of the index are formed without sign."""
    src = open(os.path.join(ROOT, "pyscf-forge_b200", "csrc", "transform_tile.cuh")).read()
    uses = re.findall(r"u\[(.*?)\];", src)
    assert uses
    for use in uses:
        for product in re.findall(r"\S+ \* \S+", use):
            assert product.count("(uint32_t)") == 2, product
