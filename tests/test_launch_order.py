"""Kernels of one stream run one after the other: no launch may start before the one ahead of it has ended."""
from pathlib import Path

PKG = Path(__file__).resolve().parent.parent / "aboleth_b200"


def test_no_kernel_is_launched_ahead_of_its_predecessor():
    """A kernel that starts early holds threads, registers, shared and tensor memory while it waits for the one
    ahead, in a wait without a limit (``griddepcontrol.wait``).  The exchange kernels size their grids by what an
    otherwise empty device holds, and their CTAs wait for one another, so what a waiting kernel of another stream holds
    can keep part of such a grid out."""
    early = ("ProgrammaticStreamSerialization", "ProgrammaticEvent", "griddepcontrol", "cudaGridDependencySynchronize",
             "cudaTriggerProgrammaticLaunchCompletion")
    suffixes = (".cu", ".cuh", ".cpp", ".hpp", ".h")
    sources = [p for d in ("csrc", "include") for p in (PKG / d).rglob("*") if p.suffix in suffixes]
    assert len(sources) > 20
    found = [f"{p.relative_to(PKG)}: {word}" for p in sources for word in early if word in p.read_text()]
    assert not found, "\n".join(found)
