"""Rotation, of rows that a trained model is applied to, of rows of any width and magnitude: widths at the edges of what the conversion to fp16 halves holds in registers, rows that
16-byte loads cannot address, row counts around a tile and around one tile per pair of SMs."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,d", [(1, 33), (130, 50), (255, 127), (257, 129), (300, 255), (140, 257), (600, 511), (300, 513), (300, 770), (256, 1_025), (130, 1_537), (70, 2_051),
                                 (520, 132), (260, 516), (130, 1_028), (100, 1_540), (19_200, 128), (18_945, 260)])
def test_rows_of_any_width_and_magnitude(n, d):
    import superkmeans_b200 as skm

    rng = np.random.default_rng(n + d)
    x = rng.standard_normal((n, d), dtype=np.float32) * (10.0 ** rng.uniform(-25, 25, (n, 1))).astype(np.float32)
    x[n // 2] = 0
    m = rng.standard_normal((d, d), dtype=np.float32) * (10.0 ** rng.uniform(-3, 3, (d, 1))).astype(np.float32)
    got = skm.engine.rotate(m, x, to_assign=True)
    want = x.astype(np.float64) @ m.T.astype(np.float64)
    # 22 bits of either factor; 64 terms one after the other in an accumulator that truncates, then fp32
    scale = np.linalg.norm(x.astype(np.float64), axis=1)[:, None] * np.linalg.norm(m.astype(np.float64), axis=1)
    assert (np.abs(got - want) <= 3e-6 * scale).all()


@pytest.mark.parametrize("d", [33, 50, 57, 63, 66, 101, 133, 258, 355, 770, 1_023, 64, 132, 384, 1_024])
def test_no_further_from_64_bits_than_the_rotation_of_a_training(d):
    import superkmeans_b200 as skm

    rng = np.random.default_rng(d)
    x, m = rng.standard_normal((2_000, d), dtype=np.float32), np.linalg.qr(rng.standard_normal((d, d)))[0].astype(np.float32)
    want = x.astype(np.float64) @ m.astype(np.float64).T
    mine, training = (np.sqrt(((skm.engine.rotate(m, x, to_assign=to_assign) - want) ** 2).mean()) for to_assign in (True, False))
    assert mine <= 1.01 * training   # (the same kernel for narrow odd rows; else a hundredth for the sampling of 2000 rows)
