"""The library's streams do not wait for the default stream, so a clear or an
upload there is ordered with nothing that runs on them. Read from the sources:
cudaMemset and host-to-device cudaMemcpy appear only in functions that wait for
the whole device before they return, or that launch on the default stream too."""
import glob
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "rhybrid_b200", "csrc")
# each with the text that makes it safe
ALLOWED = {"rhgpu_create": "cudaDeviceSynchronize", "rhgpu_dn_create": "cudaDeviceSynchronize",
           "f32Init": "cudaDeviceSynchronize", "rhgpu_neutral_density": "k_np_eval<<<blocks1d(n, 128), 128>>>"}
CALL = re.compile(r"\bcudaMemset\s*\(|\bcudaMemcpy\s*\([^;]*cudaMemcpyHostToDevice")


def functions(text):
    """(name, body) of every function that starts in column 0."""
    for m in re.finditer(r"^[A-Za-z][\w:*& <>,]*?[ *&](\w+)\([^;{}]*\)\s*\{\n", text, re.M):
        end = text.find("\n}", m.end())
        yield m.group(1), text[m.end():end]


def test_no_unordered_clear_or_upload():
    seen = 0
    for path in sorted(glob.glob(os.path.join(CSRC, "*.cu")) + glob.glob(os.path.join(CSRC, "*.h"))):
        text = open(path).read()
        inside = 0
        for name, body in functions(text):
            n = len(CALL.findall(body))
            inside += n
            if n:
                assert name in ALLOWED and ALLOWED[name] in body, (os.path.basename(path), name)
        assert inside == len(CALL.findall(text)), (os.path.basename(path), "a call outside the functions that were read")
        seen += inside
    assert seen >= 4   # the allowed ones were found
