"""What belongs to a device is kept per device: a process may launch on several, from several threads."""
import re
from pathlib import Path

CSRC = Path(__file__).resolve().parents[1] / "ksa_b200" / "csrc"


def test_launchers_keep_no_flag_or_count_of_the_first_device():
    for f in sorted(CSRC.glob("*.cu")):
        text = re.sub(r"//[^\n]*", "", f.read_text())
        assert "cudaFuncSetAttribute" not in text, f.name                # raise_smem_limit, once per device
        assert "cudaDevAttrMultiProcessorCount" not in text or f.name == "host.cu", f.name       # sm_count
