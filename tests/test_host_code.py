"""The library's host code without a GPU: its objects run on a stand-in for the CUDA runtime (tests/emu/fake_cudart.cpp)
whose device memory is host memory and whose kernels do nothing."""
import hostcode
import pytest


@pytest.fixture(scope="module")
def driver(tmp_path_factory):
    return hostcode.link(tmp_path_factory.mktemp("host") / "host", ["host_driver.cpp"])


def test_a_call_after_a_refused_call(driver):
    assert hostcode.run(driver, "after") == 0


def test_null_buffers_are_refused(driver):
    """A null stack, table or output is an error of the call, as the runtime reports it, for the entry points whose
    pageable copies go through the pinned ring too."""
    assert hostcode.run(driver, "null") == 0


def test_forked_child_exits(driver):
    """A child process forked after the library has copied with helper threads ends with its own exit code."""
    assert hostcode.run(driver, "fork") == 0


def test_second_device(driver):
    """A process that calls the library with one device current and then with another: the kernels that take more than
    48 KB of shared memory are allowed it on both."""
    assert hostcode.run(driver, "devices") == 0


def test_kept_scratch_makes_room(driver):
    """A device with little memory left: scratch kept from an earlier call does not make a later call fail."""
    assert hostcode.run(driver, "scratch") == 0


@pytest.mark.parametrize("budget, slots, chunks", [("8", "1", 9), ("40", "1", 5), ("76", "2", 5)])
def test_chunks_of_a_budget(driver, monkeypatch, budget, slots, chunks):
    """Budgets in MB at which nine 256 x 256 frames come as single frames, and as 1, 2, 3, 2, 1 (three per chunk, the first
    chunk split and the end shrinking)."""
    monkeypatch.setenv("PTB_WORKSPACE_MB", budget)
    monkeypatch.setenv("PTB_CHUNK_SLOTS", slots)
    assert hostcode.run(driver, "chunks", str(chunks)) == 0
