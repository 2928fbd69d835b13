"""What a push step loads of its predecessor's output, by the source: an overlapped
step (programmatic stream serialization) is resident while the step before it
writes, so the non-coherent path, defined for memory that is read-only as long as
the kernel runs, may serve only what no step writes. (The fault would show, if at
all, as a rare stale value, so it is looked for in the text.)"""
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "droplet_gb300", "csrc")


def kernel_text():
    """step_push.cu without comments, and without phi_range, which is never overlapped."""
    text = open(os.path.join(CSRC, "step_push.cu")).read()
    text = re.sub(r"//[^\n]*", "", text)
    at = text.index("phi_range(const FastArgs a)")
    end = text.index("\n}\n", at)
    return text[:at] + text[end:]


def test_steps_load_state_coherently():
    text = kernel_text()
    assert "griddepcontrol.wait" in text  # steps overlap: the rule applies
    assert not re.search(r"\.nc\b", text)
    assert "ldu.global" not in text
    constant = {"force", "modes", "twx", "twy", "twz"}
    for arg in re.findall(r"__ldg\(([^;]*?)\)", text):
        name = re.match(r"\s*(?:pa\.)?a\.(\w+)", arg)
        assert name and name.group(1) in constant, arg
