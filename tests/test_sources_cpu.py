"""Rules that the kernels' sources keep on every machine. Loads into several CTAs at once (the cluster
form of the bulk copies) are for programs that use one GPU only; this library also runs on
every rank of programs that use several, so no source names the form."""
import os

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "qtnh_gb300", "csrc")


def test_no_source_copies_into_several_ctas():
    word = "multi" + "cast"
    for name in sorted(os.listdir(CSRC)):
        with open(os.path.join(CSRC, name)) as f:
            assert word not in f.read(), name
