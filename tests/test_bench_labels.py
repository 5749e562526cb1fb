"""The roofline line of bench.py names the kernels that the F stage of a form launches."""
import bench


def test_f_kernels():
    w2 = bench.WORKLOADS["cfg2"]                  # 64 signals
    w4 = dict(bench.WORKLOADS["cfg1"], nant=256)  # 512
    names = {k: bench.f_kernel(*k[:2], w) for k, w in {
        (0, 1, 64): w2, (1, 1, 64): w2, (1, 3, 64): w2, (2, 1, 64): w2, (0, 1, 512): w4, (1, 1, 512): w4, (2, 1, 512): w4}.items()}
    has = {k: [n for n in ("k_fpair", "k_fscalar", "k_kmajor", "k_ftc32") if n in v] for k, v in names.items()}
    assert has == {(0, 1, 64): ["k_fpair"], (1, 1, 64): ["k_fpair"], (1, 3, 64): ["k_ftc32"], (0, 1, 512): ["k_fpair"],
                   (2, 1, 64): ["k_fscalar", "k_kmajor"], (1, 1, 512): ["k_fpair", "k_kmajor"],
                   (2, 1, 512): ["k_fscalar", "k_kmajor"]}
