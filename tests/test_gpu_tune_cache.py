"""Measured MSM window widths saved and loaded across contexts (nkr_b200_tune_save /
nkr_b200_tune_load): a loaded context reports the saved width and time without
measuring again; files of another device or of another format are refused."""
import pytest

import nkr_b200 as nk

pytestmark = pytest.mark.gpu


def test_tune_cache_round_trip(tmp_path):
    path = tmp_path / "tune.txt"
    a = nk.Context(0)
    c, ms = a.tune_msm(1 << 14)
    a.tune_save(path)
    a.close()
    text = path.read_text()
    assert text.startswith("nkr-b200-tune 1\n") and "msm 14 %d " % c in text
    b = nk.Context(0)
    assert b.tune_load(path) >= 1
    c2, ms2 = b.tune_msm(1 << 14)
    assert c2 == c and abs(ms2 - ms) < 1e-3     # the loaded entry, not a new measurement
    b.close()


def test_tune_cache_refuses_foreign_files(tmp_path):
    ctx = nk.Context(0)
    other = tmp_path / "other.txt"
    other.write_text("nkr-b200-tune 1\ndevice Some Other GPU\nsms 7\nmsm 14 12 1.0\n")
    with pytest.raises(nk.B200Error):
        ctx.tune_load(other)
    junk = tmp_path / "junk.txt"
    junk.write_text("not a tuning file\n")
    with pytest.raises(nk.B200Error):
        ctx.tune_load(junk)
    ctx.close()


def test_g2_bases_take_the_width_of_fewer_points():
    """Resident G2 bases take the tuned G1 width of the smallest tuned size up to 2^12 points,
    of half of the points up to 2^15, of a quarter up to 2^19 and of all of them beyond; with
    tuning off the model's.  One run each gives the sum of the points."""
    import numpy as np
    import oracle as O
    ctx = nk.Context(0)
    gen = O.Oracle().g2_generator()
    one = O.affine_to_jac(2, gen[None])
    sizes = [(600, 600), (1024, 1024), (1025, 1024), (4096, 1024), (4097, 2049), (1 << 15, 1 << 14),
             ((1 << 15) + 1, (1 << 13) + 1), (1 << 17, 1 << 15), ((1 << 19) + 1, (1 << 19) + 1)]
    for tune in (True, False):
        ctx.set_autotune(tune)
        for n, like in sizes[:-1] if not tune else sizes:
            b = nk.MsmBases(ctx, 2, np.tile(one, (n, 1)))
            got, _ = b.run(np.tile(O.fr_mont(1), (n, 1)))
            width = b.stats()["window_bits"]
            b.free()
            assert width == ctx.tune_msm(like if tune else n)[0], (n, tune)
            assert np.array_equal(got[:16], O.Oracle().mul_affine(2, gen, O.fr_mont(n))), n
    ctx.close()
