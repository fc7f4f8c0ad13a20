"""What the fragment cache needs to be imported: the C ABI, not the torch binding (which it loads when it first launches)."""
import os
import subprocess
import sys

ROOT = os.path.abspath(os.path.join(os.path.dirname(__file__), ".."))


def test_the_cache_can_be_imported_without_the_torch_binding():
    code = ("import os, sys\n"
            "exists = os.path.exists\n"
            "os.path.exists = lambda p: not str(p).endswith('hogatt.abi3.so') and exists(p)\n"
            "import inference_lib_b200.cache as cache\n"
            "assert cache.FragmentCache\n"
            "try:\n"
            "    import inference_lib_b200.attention\n"
            "except ImportError as e:\n"
            "    assert 'hogatt.abi3.so' in str(e)\n"
            "else:\n"
            "    sys.exit('the binding was found after all')\n")
    r = subprocess.run([sys.executable, "-c", code], cwd=ROOT, capture_output=True, text=True)
    assert r.returncode == 0, r.stdout + r.stderr
