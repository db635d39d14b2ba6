"""The binding's component record (a ctypes structure and the numpy record that proxy_components fills) against the header's
dsg_component, compiled: size, and every field's place."""
import subprocess

import dsgpu
import libs


def test_component_record(tmp_path):
    names = dsgpu.COMPONENT.names
    src, exe = tmp_path / "layout.c", tmp_path / "layout"
    src.write_text('#include <stddef.h>\n#include <stdio.h>\n#include "dsgpu.h"\nint main(void) { printf("%zu", sizeof(dsg_component));\n'
                   + "".join(f'printf(" %zu", offsetof(dsg_component, {n}));\n' for n in names) + "return 0; }\n")
    subprocess.check_call(["gcc", "-I" + libs.ROOT + "/include", str(src), "-o", str(exe)])
    size, *at = map(int, subprocess.check_output([str(exe)]).split())
    assert dsgpu.COMPONENT.itemsize == size == dsgpu.C.sizeof(dsgpu.Component)
    assert [dsgpu.COMPONENT.fields[n][1] for n in names] == at == [getattr(dsgpu.Component, n).offset for n in names]
