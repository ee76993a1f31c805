"""Host code plans for the current device: none of it asks for a device by number."""
import glob
import os
import re

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_no_attribute_of_a_device_by_number():
    asked = []
    for path in glob.glob(os.path.join(ROOT, "codesthesis_dir_gb300", "csrc*", "*")):
        for m in re.finditer(r"cuda(?:DeviceGetAttribute|GetDeviceProperties)\s*\(([^;]*)\)\s*[;)]", open(path).read()):
            if re.search(r",\s*\d+\s*$", m.group(1).split("!=")[0].rstrip(") ")):
                asked.append((os.path.basename(path), m.group(0)))
    assert not asked, asked
