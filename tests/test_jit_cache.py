"""Reuse of models generated for run-time compilation."""
from __future__ import annotations

import json

from goss_b200 import compilemodule
from goss_b200.codegen.odeparse import parse_ode_text
from goss_b200.codegen.variant import GENERATOR_VERSION
from goss_b200.models import variant_dirs

GATES = "states({})\n{}".format(", ".join(f"x{i}=0.1" for i in range(10)),
                                "".join(f"dx{i}_dt = -{i + 1}.0*x{i} + exp(-x{(i + 1) % 10})\n" for i in range(10)))


def test_text_of_another_generator_version_is_written_again(tmp_path, monkeypatch):
    monkeypatch.setattr(compilemodule, "JIT_DIR", tmp_path)
    monkeypatch.setattr(compilemodule, "load_variant", lambda vdir: vdir)
    vdir = compilemodule.jit(parse_ode_text(GATES, "cache_gates"))
    device, meta = vdir / "device.cuh", vdir / "model.json"
    text = device.read_text()
    assert "linear_group" in text and json.loads(meta.read_text())["generator_version"] == GENERATOR_VERSION
    # as the version before the row groups left it
    device.write_text("\n".join(x for x in text.split("\n") if "_group(int" not in x))
    meta.write_text(json.dumps({**json.loads(meta.read_text()), "generator_version": "8"}))
    assert compilemodule.jit(parse_ode_text(GATES, "cache_gates")) == vdir
    assert device.read_text() == text and json.loads(meta.read_text())["generator_version"] == GENERATOR_VERSION
    # and the current one is left alone
    monkeypatch.setattr(compilemodule, "write_variant", None)
    assert compilemodule.jit(parse_ode_text(GATES, "cache_gates")) == vdir


def test_shipped_models_are_of_this_version():
    assert all(json.loads((d / "model.json").read_text())["generator_version"] == GENERATOR_VERSION
               for d in variant_dirs())
