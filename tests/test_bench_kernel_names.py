"""CPU: the bench names the kernels that a context took, not those that its size would suggest."""
import pytest

from test_bench_contract import load_bench


class Context:
    def __init__(self, group, viscous=0):
        self.group, self.viscous = group, viscous

    def kernel_group(self, viscous=False):
        return self.viscous if viscous else self.group


@pytest.mark.parametrize("precision,group,viscous,mu,face", [
    ("fp64", 8, 0, 0.0, "face_flux_rows8"), ("fp64", 3, 0, 0.0, "face_flux_tc"), ("fp64", 1, 0, 0.0, "face_flux_fp64"),
    ("fp64", 3, 8, 0.1, "visc_face_rows8"), ("fp64", 3, 1, 0.1, "face_flux_tc"),
    ("mixed", 16, 0, 0.0, "face_flux_mixed16"), ("mixed", 3, 8, 0.1, "face_flux_mixed")])
def test_names_follow_the_context(precision, group, viscous, mu, face):
    b = load_bench()
    names = b.kernel_names(precision, "two-launch", Context(group, viscous), mu)
    assert names[0] == face
    for name in names.values():
        assert b.kernel_bytes(name, 3, 6 * 12 ** 3, 12 * 12 ** 3, 24) > 0
    kt = {0: (2.0, 3), 1: (1.0, 3)}
    r = b.make_roofline(kt, precision, "two-launch", 3, 6 * 12 ** 3, 12 * 12 ** 3, 24, 20, "tgv", mu, Context(group, viscous))
    assert r["kernel"] == face
