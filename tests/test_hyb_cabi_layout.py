"""The mirrors in tests/hyb_cabi.py against the header, as the C compiler lays it out."""
import os
import subprocess

import hyb_cabi as H

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_structs_match_the_header(tmp_path):
    src = ['#include <stdio.h>', '#include "tha_hybrid.h"', "int main(void) {"]
    want = []
    for s in H.STRUCTS:
        src.append('printf("%%zu\\n", sizeof(%s));' % s.__name__)
        want.append(H.C.sizeof(s))
        for f, _ in s._fields_:
            src.append('printf("%%zu\\n", offsetof(%s, %s));' % (s.__name__, f))
            want.append(getattr(s, f).offset)
    (tmp_path / "a.c").write_text("\n".join(src + ["return 0; }"]))
    subprocess.check_call(["gcc", "-I", os.path.join(ROOT, "include"), "-o", str(tmp_path / "a"), str(tmp_path / "a.c")])
    assert [int(x) for x in subprocess.check_output([str(tmp_path / "a")]).split()] == want
