"""How many output pairs a thread of a wavelet pass owns (host code, runtime
faked, 152 SMs): four where that is faster by the measurements beside the rule,
one elsewhere."""
from host_cuda import host_cuda  # noqa: F401

HAAR, BIOR13, BIOR22, BIOR24, BIOR31 = range(5)
# (h, w), filter -> pairs in the passes along x and along y
WANT = [((256, 256), BIOR22, 1), ((512, 512), BIOR22, 4), ((512, 512), BIOR24, 4), ((512, 512), BIOR13, 1),
        ((512, 512), HAAR, 1), ((640, 640), BIOR22, 1), ((640, 640), BIOR24, 1), ((768, 768), BIOR22, 4),
        ((768, 768), BIOR31, 1), ((1024, 1024), HAAR, 1), ((1024, 1024), BIOR22, 1), ((1024, 1024), BIOR24, 1),
        ((2048, 2048), HAAR, 1), ((2048, 2048), BIOR13, 4), ((2048, 2048), BIOR22, 4), ((2048, 2048), BIOR31, 1),
        ((4096, 4096), HAAR, 4), ((4096, 4096), BIOR31, 4),
        # the shapes of tests/test_gpu_wavelet_pairs.py
        ((470, 490), BIOR22, 4), ((470, 490), BIOR24, 4), ((1524, 756), HAAR, 4), ((1524, 756), BIOR13, 4),
        ((1524, 756), BIOR31, 4)]

SCRIPT = r"""
import re
result = []
for (h, w), f in %r:
    data, temp = cells((h, w), 8), cells((h, w), 8)
    log()
    rc = lib.pg_wavelet_fwt_2d(0, f, f, data, h, w, 1, temp, None) or lib.pg_wavelet_ifwt_2d(0, f, f, data, h, w, 1, temp, None)
    result.append((rc, [[int(v) for v in re.search(r"k_w(?:down|up)_[xy]ILi(\d)ELi(\d)E", k).groups()] for k in kernels()]))
    keep.clear()
"""


def test_pairs(host_cuda):  # noqa: F811
    got = host_cuda(SCRIPT % [(s, f) for s, f, _ in WANT])
    for (shape, f, pairs), (rc, passes) in zip(WANT, got):
        assert rc == 0 and passes == [[f, pairs]] * 4, (shape, f, passes)
