"""What the build leaves behind: an installed package holds every built file, and a module built against another torch or Python is
built anew."""
import re
import tomllib
from pathlib import Path

from turboquant_b200 import build

ROOT = Path(__file__).resolve().parent.parent


def test_package_data_covers_the_built_files():
    patterns = tomllib.loads((ROOT / "pyproject.toml").read_text())["tool"]["setuptools"]["package-data"]["turboquant_b200"]
    packaged = {path for pattern in patterns for path in build.PKG.glob(pattern)}
    build.build()
    for built in (build.LIB, build.NATIVE, build.NATIVE_SRC):
        assert built in packaged, built


def test_the_native_module_is_bound_to_torch_and_python(monkeypatch, tmp_path):
    build.build()
    assert not build._native_stale()
    monkeypatch.setattr("torch.__version__", "0.0.0")
    assert build._native_stale()
    monkeypatch.undo()
    monkeypatch.setattr(build, "NATIVE_STAMP", tmp_path / "none")      # a module of before the stamp
    assert build._native_stale()


def test_no_kernel_gives_up_on_a_copy_in_silence():
    """Every bounded wait for a copy, where it runs out, raises a status or counts a fault before its warp returns; a copy that is lost cannot be made on
    purpose, so this reads the source."""
    csrc = Path(build.__file__).parent / "csrc"
    seen = 0
    for path in sorted(csrc.glob("*.cu*")):
        text = path.read_text()
        for at in re.finditer(r"\bmbar_wait\(&", text):
            seen += 1
            handler = text[at.start():at.start() + 400]
            assert "copy_lost(" in handler or "abort_flag = 1" in handler, f"{path.name}: {handler[:120]}"
    assert seen >= 6
