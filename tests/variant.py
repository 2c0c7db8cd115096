"""Programs run on the library with one of its files compiled with other
build knobs, in a process of their own."""
import glob
import importlib.util
import os
import subprocess
import sys

from conftest import PKG, ROOT


def run_with_variant(tmp_path, source, knobs, program, *args):
    """Compiles csrc/`source` with `knobs`, links it with the other objects of the
    built library, and runs `program` (text) with the path of the result and `args`;
    the program has to print ok."""
    spec = importlib.util.spec_from_file_location("_lpgpu_build", os.path.join(PKG, "build.py"))
    recipe = importlib.util.module_from_spec(spec)
    spec.loader.exec_module(recipe)
    name = os.path.splitext(source)[0] + ".o"
    obj, so = str(tmp_path / name), str(tmp_path / "liblpgpu_variant.so")
    subprocess.run([recipe.nvcc()] + recipe.ARCH + recipe.NVCC_FLAGS + knobs +
                   ["-c", os.path.join(recipe.CSRC, source), "-o", obj], check=True)
    others = [o for o in glob.glob(os.path.join(recipe.BUILD, "*.o")) if os.path.basename(o) != name]
    subprocess.run([recipe.nvcc()] + recipe.ARCH + ["-shared", "-o", so, obj] + others + ["-cudart", "static"], check=True)
    r = subprocess.run([sys.executable, "-c", program, so] + list(args), capture_output=True, text=True, timeout=300,
                       env=dict(os.environ, PYTHONPATH=os.pathsep.join([PKG, ROOT])))
    assert r.returncode == 0 and r.stdout.strip() == "ok", r.stdout + r.stderr
