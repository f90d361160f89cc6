"""The quotients, reciprocals and roots of rod_fast.cuh round as IEEE division
and square root do (GPU), bit for bit against NumPy's.

A correction by the residual leaves out a term below 2^-100 of the result, so
what could go wrong are arguments whose result lies that near to the middle of
two doubles.  They are listed or constructed here; random ones never meet them."""
import ctypes
import subprocess

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# Significands D (53 bits) with D M = 2^106 - k, |k| <= 20, for an odd M of 54
# bits: 1 / D is within 2^-101 of a tie (found by factoring 2^106 - k)
NEAR_TIES = np.array([
    4526458347800502, 4543885306550786, 4619723575576654, 4663060627120798, 4691463364816860, 4694365760365840,
    4696637379339158, 4713086531278084, 4732570949897334, 4764758390727204, 4797136447748302, 4799436974858658,
    4826740803455362, 4853175449558581, 4889509067008578, 5017593869129758, 5059465667261026, 5078160416645382,
    5113735303349264, 5146971002709136, 5147049539853168, 5161381560812848, 5161460317846224, 5227109417592368,
    5259296635906338, 5276938686109394, 5298352502788820, 5316991813459108, 5322981989608814, 5349226260991312,
    5359079149933474, 5384033562998736, 5384074640541744, 5384724193248396, 5433304946044738, 5440503800133692,
    5481939640292082, 5497283260653072, 5527402342438382, 5532337980645058, 5584820410479762, 5633797035358998,
    5681288978402960, 5778203295494220, 5813097674954626, 5852518495683566, 5947121809636240, 6004799503160660,
    6015585163436338, 6028126993990242, 6080991238998918, 6195114542651238, 6223412073831755, 6258053705355746,
    6259525790675524, 6260414481236258, 6428029221663302, 6457373739988182, 6468322654107666, 6525673443791140,
    6530993532304592, 6583997076838894, 6628645658878754, 6629242916101340, 6636062006759376, 6743444718440206,
    6762858185200722, 6789477085927202, 6817518320890736, 6825891612808598, 6836844636365422, 6861827417050864,
    6861932121026832, 6877576621274544, 7022242040581488, 7052061190152272, 7067989545731856, 7111558598256016,
    7118995707580124, 7120733955830052, 7131469634928688, 7131524043309008, 7143133470683622, 7177928720498256,
    7205759189044432, 7209683550988788, 7210714368219586, 7262274947386576, 7302143716234066, 7331062497459854,
    7341008258195058, 7367710770432518, 7440678027627698, 7492481886289796, 7502829227184258, 7571806663240402,
    7637721365894914, 7857326865746386, 7923715856877378, 7941263984545340, 7943203006394820, 7966213734168822,
    7997569094099302, 8042426583074580, 8240382507728326, 8263449212651198, 8273878955596112, 8340967600624526,
    8413745725510706, 8414153661196722, 8480179861092514, 8573369051977618, 8599630430979522, 8614211686276086,
    8691914294970288, 8712776903364457, 8716460134775102, 8837852221345158, 8852837397806754, 8901779882296592,
    8952924378397104, 8974540322080660, 9002296740580796, 9007199120523265, 9007199254740989, 9007199254740991,
], dtype=np.float64) / 2.0 ** 52


@pytest.fixture(scope="module")
def probe(tmp_path_factory):
    import os

    from elasticapp_b200 import build as b

    out = str(tmp_path_factory.mktemp("probe") / "rod_fast_probe.so")
    src = os.path.join(os.path.dirname(os.path.abspath(__file__)), "rod_fast_probe.cu")
    subprocess.run([b.nvcc()] + b.common_flags() + ["-Xcompiler", "-fvisibility=default", "-shared", src, "-o", out],
                   check=True)
    lib = ctypes.CDLL(out)

    def run(op, a, c=None):
        a = np.ascontiguousarray(a, dtype=np.float64).ravel()
        c = a if c is None else np.ascontiguousarray(c, dtype=np.float64).ravel()
        o, o2 = np.empty_like(a), np.empty_like(a)
        ptr = [ctypes.c_void_p(z.ctypes.data) for z in (a, c, o, o2)]
        assert lib.rod_fast_probe(op, a.size, *ptr) == 0
        return o, o2

    return run


def ulps(x, k):
    return (x.view(np.int64) + k).view(np.float64)


def exponents(a, low, high):
    """a at every exponent from low to high."""
    return np.ldexp(np.asarray(a)[:, None], np.arange(low, high + 1)).ravel()


def significands():
    """Random, and next to powers of two."""
    near = np.concatenate([ulps(np.full(9, x), np.arange(-4, 5)) for x in (1.0, 2.0)])
    return np.concatenate([np.random.default_rng(91).uniform(1.0, 2.0, 4096), near[(near >= 1.0) & (near < 2.0)]])


def test_reciprocals_next_to_ties(probe):
    d = exponents(NEAR_TIES, -400, 399)
    np.testing.assert_array_equal(probe(0, d)[0], 1.0 / d)
    y = 1.0 / NEAR_TIES
    # a start off by half an ulp is the double on either side of the tie
    above = np.array([int(D * 2.0 ** 52) * int(v * 2.0 ** 53) < 2 ** 105 for D, v in zip(NEAR_TIES, y)])  # 1 / D > y
    for other in (y, np.where(above, ulps(y, 1), ulps(y, -1))):
        np.testing.assert_array_equal(probe(1, NEAR_TIES, other)[0], y)
    for k in range(-16, 17):
        np.testing.assert_array_equal(probe(2, NEAR_TIES, ulps(y, k))[0], y)


def test_lengths_next_to_ties(probe):
    # every square whose root rounds to such a divisor
    z = np.concatenate([ulps(NEAR_TIES ** 2, k) for k in range(-4, 5)])
    # the squares whose roots are nearest to a tie: M^2 = Z 2^s - k, k = 7 and 23
    z = np.concatenate([z, [6114741795106786 / 2.0 ** 51, 8233674359446949 / 2.0 ** 52, 5888295035175849 / 2.0 ** 51]])
    z = np.ldexp(z[:, None], np.arange(-398, 397, 2)).ravel()
    length, inverse = probe(4, z)
    np.testing.assert_array_equal(length, np.sqrt(z))
    np.testing.assert_array_equal(inverse, 1.0 / np.sqrt(z))


def test_quotients_next_to_ties(probe):
    rng, a, b = np.random.default_rng(92), [], []
    divisors = [int(x) | (1 << 52) | 1 for x in rng.integers(0, 1 << 52, 4000)] + [int(D * 2.0 ** 52) | 1 for D in NEAR_TIES]
    for D in divisors:
        inverse = pow(D, -1, 1 << 54)
        for k in (1, -1, 2, -2, 3, -3, 4, -4, 5, -5):
            for s in (53, 54):  # A 2^s = D M + k with an odd M of 54 bits: A / D within 2^-106 of a tie
                M = (-k * inverse) % (1 << s) + ((1 << 53) if s == 53 else 0)
                A = (D * M + k) >> s
                if M % 2 and M > 1 << 53 and 1 << 52 <= A < 1 << 53 and (s == 53) == (A >= D):
                    a.append(A / 2.0 ** 52)
                    b.append(D / 2.0 ** 52)
    a, b = np.array(a), np.array(b)
    assert a.size > 10000
    for e in (-399, -1, 0, 1, 399):
        c = np.ldexp(b, e)
        np.testing.assert_array_equal(probe(3, a, c)[0], a / c)


def test_the_whole_range(probe):
    x = exponents(significands(), -400, 399)
    np.testing.assert_array_equal(probe(0, x)[0], 1.0 / x)
    length, inverse = probe(4, x)
    np.testing.assert_array_equal(length, np.sqrt(x))
    np.testing.assert_array_equal(inverse, 1.0 / np.sqrt(x))
    a = np.random.default_rng(93).permutation(x)
    np.testing.assert_array_equal(probe(3, a, x)[0], a / x)
    # outside it the plain operations
    x = np.concatenate([exponents([1.0, 1.7], -1074, -401), exponents([1.0, 1.7], 400, 1023), [0.0, np.inf]])
    with np.errstate(divide="ignore"):
        np.testing.assert_array_equal(probe(4, x)[0], np.sqrt(x))
        np.testing.assert_array_equal(probe(4, x)[1], 1.0 / np.sqrt(x))
