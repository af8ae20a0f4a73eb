"""What the learner's head plans its backward by, on the CPU."""
import pytest
import torch

from pipelinerl_b200.learner_model import _NativeHead


@pytest.mark.parametrize("M,chunk", [(0, 64), (1, 64), (64, 64), (3071, 3072), (4096, 4096), (4097, 2112), (8192, 4096), (8193, 2752), (16383, 4096)])
def test_rows_of_a_chunk(M, chunk):
    """Up to 4096 rows at once, more in equal chunks of whole k-blocks."""
    assert _NativeHead._chunk_rows(M) == chunk and -(-max(M, 1) // chunk) == max(1, -(-M // 4096))


@pytest.mark.parametrize("M,V,chunk,free_gb,rows", [(256, 152064, 256, 100, 0), (257, 152064, 320, 100, 257), (3071, 152065, 3072, 100, 0), (3071, 152064, 3072, 100, 3071),
                                                    (3071, 152064, 3072, 7, 0), (8192, 152064, 4096, 11, 4096), (8192, 152064, 4096, 9, 0), (8192, 152064, 4096, 21, 8192)])
def test_rows_whose_logits_are_kept(monkeypatch, M, V, chunk, free_gb, rows):
    """A quarter of the free memory (what the allocator holds unused is free), all rows or whole chunks; none for few rows or odd vocabularies."""
    monkeypatch.setattr(torch.cuda, "mem_get_info", lambda dev: ((free_gb - 3) * 10 ** 9, 0))
    monkeypatch.setattr(torch.cuda, "memory_reserved", lambda dev: 13 * 10 ** 9)
    monkeypatch.setattr(torch.cuda, "memory_allocated", lambda dev: 10 ** 10)
    assert _NativeHead._rows_to_keep(M, V, None, chunk) == rows


@pytest.mark.parametrize("rows", [1, 3, 8])
def test_kept_logits_of_a_batch_share_a_quarter(monkeypatch, rows):
    """Row after row of a batch, each with less memory left: together they take no more than a quarter of what was free before the first."""
    free, held, M, V = 40 * 10 ** 9, 0, 4096, 152064
    monkeypatch.setattr(torch.cuda, "mem_get_info", lambda dev: (free - held, 0))
    monkeypatch.setattr(torch.cuda, "memory_reserved", lambda dev: held)
    monkeypatch.setattr(torch.cuda, "memory_allocated", lambda dev: held)
    for _ in range(rows):
        held += 4 * V * _NativeHead._rows_to_keep(M, V, None, M, held)
    assert held == 4 * V * M * min(rows, 4) <= free // 4
