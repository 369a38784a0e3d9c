"""pysa_gb_set_block_round_limit: its default can be set again."""


def test_default_limit_comes_back():
    from pysa_gb300 import _lib
    lib = _lib.load()
    shapes = [(n, c) for n in (64, 512, 513, 1024, 1025, 2048)
              for c in (1, 32, 33, 128)]
    # 4 where a block's sub-blocks are relayed and both forms round alike
    default = [4 if n > 1024 or (n <= 512 and c <= 32) else 12
               for n, c in shapes]

    def limits():
        return [lib.pysa_gb_tc_round_limit(n, c) for n, c in shapes]

    try:
        for flips in (0, 4, 13, 64):
            assert lib.pysa_gb_set_block_round_limit(flips) == 0
            assert limits() == [flips] * len(shapes)
    finally:
        assert lib.pysa_gb_set_block_round_limit(12) == 0
    assert limits() == default
    assert lib.pysa_gb_tc_round_limit(63, 1) == -1
    assert lib.pysa_gb_tc_round_limit(64, 0) == -1
