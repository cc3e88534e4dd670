"""The workspace of SLIC and plane snapping (host only, no GPU)."""


def test_postprocessing_needs_no_more_than_before(svb):
    """SLIC and plane snapping: centres, windows, sums, distances, labels, lists,
    states side by side, as the library asked for before."""
    lib = svb._lib.load()
    up = lambda n: (n + 255) // 256 * 256
    for W in list(range(1, 40)) + [160, 450]:
        for H in list(range(1, 40, 3)) + [120, 375]:
            for step in (1, 2, 5, 12, 30, 100):
                N, nc = W * H, max(1, lib.sv_slic_count(W, H, step))
                before = (256 + up(40 * nc) + up(16 * nc) + up(48 * nc) + 2 * up(8 * N) +
                          5 * up(4 * N) + 256 + 3 * up(4 * nc) + up(4 * (nc + 1)) + up(N))
                assert lib.sv_postproc_workspace_size(W, H, step) <= before, (W, H, step)
