"""Which transform each axis length gets, without a GPU: every length has a valid one, and
every compiled one is some length's."""
import line_plans as L


def test_every_length_has_a_transform():
    for n, (direct, variant, n1, n2) in L.plans().items():
        assert variant in ((16, 24, 32, 64) if direct else (0,))
        if direct:
            assert n1 * n2 == n and n1 <= n2 <= variant
            assert (variant == 64) == (n > 1024)
        else:
            assert (n1, n2) in L.compiled_chirps()
            # the shortest that holds the linear convolution
            assert n1 * n2 == min(a * b for a, b in L.compiled_chirps() if a * b >= 2 * n - 1)


def test_every_compiled_convolution_is_used():
    assert {p[2:] for p in L.plans().values() if not p[0]} == L.compiled_chirps()


def test_edge_lengths_cover_all_transforms():
    every = {(d, v, a) for d, v, a, b in L.plans().values()} | \
        {(d, v, -b) for d, v, a, b in L.plans().values()}
    edge = [L.plans()[n] for n in L.edge_lengths()]
    got = {(d, v, a) for d, v, a, b in edge} | {(d, v, -b) for d, v, a, b in edge}
    assert every - got <= {(1, 16, 1), (1, 16, -1), (1, 16, -2)}  # n = 1, 2
