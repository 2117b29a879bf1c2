"""The structures that the library fills in for its callers have the size that
programs compiled against earlier headers reserved for them."""
import ctypes
import os
import subprocess

import slcs

INCLUDE = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "include")
SIZES = {"slcs_config": 64, "slcs_pair_info": 64, "slcs_plan_info": 48, "slcs_pair_desc": 32}


def test_header(tmp_path):
    src = tmp_path / "sizes.c"
    src.write_text('#include "slcs.h"\n' + "".join(f'_Static_assert(sizeof({t}) == {s}, "{t}");\n'
                                                    for t, s in SIZES.items()) + "int x;\n")
    subprocess.run(["gcc", "-c", "-I", INCLUDE, str(src), "-o", str(tmp_path / "sizes.o")], check=True)


def test_binding():
    for kind, name in ((slcs.Config, "slcs_config"), (slcs.PairInfo, "slcs_pair_info"),
                       (slcs.PlanInfo, "slcs_plan_info"), (slcs.PairDesc, "slcs_pair_desc")):
        assert ctypes.sizeof(kind) == SIZES[name]
