"""The executed FLOPs that the rates are printed with, against the MMAs of the
one-kernel forward pass counted window by window."""


def test_network_mmas():
    import learned
    flop = 10 * 14 * 128 * 32 * 16 * 2                       # layer 1: tap pairs
    for nout, z_min, z_max in ((32, 0, 9), (32, 0, 9), (16, 1, 8)):
        for w in range(10):                                  # window: input plane w
            planes = min(w + 1, z_max) - max(w - 1, z_min) + 1
            flop += 18 * 128 * nout * planes * 16 * 2        # 9 (dy, dx) x 2 halves of 32 channels
    assert learned.NET_FLOP_EXECUTED == flop
