"""The bytes that the benchmark's roofline fraction counts are those a step cannot do without."""
import bench


def test_bytes_of_a_step():
    Np, Nfp, nf, s = 220, 55, 4, 4
    step = 0
    for stage in range(5):
        step += 2 * nf * Np * s                      # q in and out
        step += (1 if stage == 0 else 2) * nf * Np * s  # res out; in, but for the first (A = 0)
        step += 4 * nf * Nfp * s + 22 * s + 4 * 4    # traces, geometry, connectivity
    assert abs(5 * bench.stage_bytes_per_element() - step) < 1e-6
