"""The network's layers may start while the kernel before them still writes their input rows (Hin). Loads that ask
for data that is read-only for the kernel's lifetime (__ldg, ld.global.nc, a const __restrict__ parameter)
are therefore not for those rows: read from the source, since no run shows it."""
import os
import re

REPO = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(REPO, "mpi-cst-fem-solver_b200", "csrc")


def test_no_read_only_loads_of_chained_rows():
    text = open(os.path.join(CSRC, "mpnn.cu")).read()
    chained = sorted(set(re.findall(r"launch_next\((k_\w+)", text)))
    assert chained == ["k_mp_layer_tc", "k_mp_layer_ws"]
    for name in chained:
        at = text.index(f"{name}(const MpLayerArgs")
        body = text[at:text.index("\n}\n", at)]
        assert "wait_previous()" in body and "Hin" in body
        for call in re.findall(r"(__ldg\(|ld\.global\.nc)([^;]*)", body):
            assert "Hin" not in call[1].split("ld_chained")[0], call
    args = text[text.index("struct MpLayerArgs"):]
    assert "__restrict__" not in args[:args.index("};")]
