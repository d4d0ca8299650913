"""Radices of the any-extent transforms, for every extent a context takes (host only).

The register kernels exist for 2 .. 13 and 16; any other radix is a prime summed
pair by pair, so a composite there costs a factor in operations though the result
is right."""
import ctypes as C

import pytest

REGISTER = set(range(2, 14)) | {16}


def _radices(n):
    from langevinfts_b200.capi import lib
    r, count = (C.c_int * 16)(), C.c_int()
    if lib().lfts_transform_radices(n, r, 16, C.byref(count)) != 0:
        return None
    return list(r[:count.value])


def _primes(n):
    out, p = [], 2
    while n > 1:
        while n % p == 0:
            out.append(p)
            n //= p
        p += 1
    return out


def test_plans_hold_register_radices_and_primes_only():
    for n in range(1, 1025):
        r, p = _radices(n), _primes(n)
        if p and p[-1] > 64:
            assert r is None, n
            continue
        prod = 1
        for x in r:
            prod *= x
        assert prod == n, (n, r)
        assert all(x in REGISTER or _primes(x) == [x] for x in r), (n, r)
        # primes above 13 innermost, where they need no twiddles
        assert [x for x in r if x > 16] == r[len(r) - sum(x > 16 for x in r):], (n, r)


@pytest.mark.parametrize("n,stages", [(16, 1), (48, 2), (75, 3), (98, 3), (105, 3), (125, 3), (169, 2), (196, 3), (220, 3), (256, 2)])
def test_number_of_stages(n, stages):
    assert len(_radices(n)) == stages


def test_refusals():
    assert _radices(0) is None and _radices(1025) is None and _radices(134) is None  # 134 = 2 x 67
