"""Contexts on different threads share the library's process-wide state: what the native sources keep for the
process is const (set up once by the language's own guard), atomic or thread-local."""
import glob
import os
import re

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
# a `static` variable, or a file-scope one by its g_ name, of a plain type
PLAIN = re.compile(r"^\s*(?:static\s+(?:inline\s+)?(?:bool|int|unsigned|float|u?int\d+_t)\s+\w+"
                   r"|(?:bool|int|unsigned|float|u?int\d+_t)\s+g_\w+)[^()]*;", re.M)


def test_no_unguarded_process_state():
    sources = [f for ext in ("cu", "cuh", "h") for f in glob.glob(os.path.join(ROOT, "mcrt_gb300", "csrc", "*." + ext))]
    assert len(sources) > 10
    found = {os.path.basename(f): PLAIN.findall(open(f).read()) for f in sources}
    assert not any(found.values()), {f: v for f, v in found.items() if v}
