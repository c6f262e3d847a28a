"""The library's build: one source, one library."""
import importlib.util
import os

import pkg


def test_no_option_lets_the_compiler_cut_the_module_by_timing():
    """-split-compile with more than one thread gave two libraries in turn, with
    other code for pass 1 and other last bits in fast arithmetic."""
    spec = importlib.util.spec_from_file_location("hosono_build", os.path.join(pkg.PKG_DIR, "build.py"))
    build = importlib.util.module_from_spec(spec)
    spec.loader.exec_module(build)
    commands = [cmd for _, _, cmd in build.jobs()]
    assert any(c.endswith("kernels.cu") for cmd in commands for c in cmd)
    for cmd in commands:
        assert not [a for a in cmd if a.lstrip("-").startswith("split-compile")]
