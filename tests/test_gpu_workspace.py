"""GPU test of a call slot's device memory: per HSP of its capacity 96 bytes, the
arrays that a call uses (two record and scope buffers, the sweep's list, and
two slots of the HSP set)."""
import pytest

from segalign_b200 import SeedFilter, build_sub_mat

pytestmark = pytest.mark.gpu


def test_bytes_per_record_of_capacity(built, monkeypatch):
    import torch
    sf = SeedFilter()
    sf.initialize_interface(1)
    sf.generate_shape_pos("12of19")
    monkeypatch.setenv("SA_SLOTS_PER_GPU", "1")
    used = []
    for cap in (1 << 20, 1 << 25):
        monkeypatch.setenv("SA_SURV_CAP", str(cap))
        sf.shutdown_processor()
        free = torch.cuda.mem_get_info()[0]
        sf.initialize_processor(False, 10_000, 19, build_sub_mat(910), 910, 3000, False)
        used.append(free - torch.cuda.mem_get_info()[0])
    monkeypatch.undo()
    sf.initialize_processor(False, 10_000, 19, build_sub_mat(910), 910, 3000, False)
    assert abs(used[1] - used[0] - 96 * ((1 << 25) - (1 << 20))) <= 8 << 20  # the allocator's granularity
