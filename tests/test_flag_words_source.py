"""The grid CG's published words carry 32 bits of data and a 32-bit flag, and a
reader takes the data when it sees the flag. That needs each word to be one 64-bit
access; a vector of 32-bit elements is several accesses in no stated order, which
no run on a device would show. The check is of the source."""
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "cfdrs_b200", "csrc")


def test_words_are_64_bit_accesses():
    text = open(os.path.join(CSRC, "grid_pcg.cu")).read()
    accesses = re.findall(r"\b(?:ld|st)\.volatile\.global\.([\w.]+)", text)
    assert len(accesses) == 2 and set(accesses) <= {"v2.b64", "v2.u64", "b64", "u64"}, accesses


def packed(bits, flag):
    return (bits & 0xFFFFFFFF) | flag << 32, bits >> 32 | flag << 32


def test_packing_round_trips():
    """The arithmetic of gp_publish and gp_read on the bit patterns where it could go wrong."""
    for bits in (0, 1, 1 << 31, 1 << 32, 0x7FF0000000000000, 0xFFF8000000000001, (1 << 64) - 1):
        for flag in (1, 2, 1 << 31, (1 << 32) - 1):
            a, b = packed(bits, flag)
            assert a >> 32 == flag and b >> 32 == flag
            assert (a & 0xFFFFFFFF | b << 32) & (1 << 64) - 1 == bits
