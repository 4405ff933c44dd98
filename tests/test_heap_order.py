"""The order of the heap's superblock hand-overs (no GPU).

The functions' own text is taken out of include/kma_device.cuh and compiled
for the host against words whose stores become visible as late as the
memory model allows: a plain store waits until a release of the same thread.
Between any two accesses another thread does the most it may with what is
visible by then."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
DEVICE = os.path.join(ROOT, "include", "kma_device.cuh")

COMMON = r"""
#include <cstdint>
#include <cstdio>
#include <cstring>
#include <functional>
#include <utility>
#include <vector>
#define __device__
#define __forceinline__ inline
static const uint32_t CLS = 3;
static uint32_t st_free(uint32_t s) { return s & 0x3fffu; }
static uint32_t st_slots(uint32_t s) { return (s >> 14) & 0x3fffu; }
static uint32_t st_class(uint32_t s) { return s >> 28; }
static uint32_t st_make(uint32_t c, uint32_t slots, uint32_t fr) { return c << 28 | slots << 14 | fr; }
static std::vector<std::function<void()>> pending; /* plain stores not yet visible */
static void land() { for (auto &f : pending) f(); pending.clear(); }
static std::function<void()> other = [] {};         /* the other thread, between accesses */
struct word {                                        /* a word stored to plainly */
	uint32_t v;
	void operator=(uint32_t x) { pending.push_back([this, x] { v = x; }); }
};
"""

FORMAT = COMMON + r"""
struct kma_heap { uint32_t cls_slots[16], cls_words[16]; word sb_home[4]; uint32_t sb_state[4]; };
static word bitmap[64];
static unsigned char *sb_addr(kma_heap *, uint32_t) { return nullptr; }
static word *bitmap_word(kma_heap *, unsigned char *, uint32_t k) { return &bitmap[k]; }
static void st_release(uint32_t *p, uint32_t v) { land(); *p = v; other(); }
static void st_relaxed(uint32_t *p, uint32_t v) { *p = v; other(); }
%s
int main(int, char **argv)
{
	uint32_t slots = atoi(argv[1]), pre_lo = atoi(argv[2]), words = (slots + 31) / 32;
	static kma_heap h;
	h.cls_slots[CLS] = slots;
	h.cls_words[CLS] = words;
	/* what an earlier incarnation left behind */
	for (uint32_t k = 0; k < words; k++)
		bitmap[k].v = k %% 2 ? 0x5a5a5a5au : 0u;
	h.sb_home[1].v = 9;
	h.sb_state[1] = st_make(CLS, slots, 0);
	std::vector<uint32_t> got;
	bool bad = false;
	/* another warp, whose hint names the superblock: takes every free slot
	 * that the state offers it */
	other = [&] {
		uint32_t n = st_class(h.sb_state[1]) == CLS ? st_free(h.sb_state[1]) : 0;
		h.sb_state[1] -= n;
		for (uint32_t i = 0; i < slots && n; i++)
			if (!(bitmap[i / 32].v >> (i %% 32) & 1)) {
				bitmap[i / 32].v |= 1u << (i %% 32);
				got.push_back(i);
				n--;
			}
		bad |= n != 0 || h.sb_home[1].v != 5;
	};
	sb_format(&h, 1, CLS, pre_lo, pre_lo, 5);
	land();
	for (uint32_t i : got) /* its slots are its own, and stay claimed */
		bad |= i >= pre_lo || !(bitmap[i / 32].v >> (i %% 32) & 1);
	printf("%%s\n", bad || got.size() != pre_lo ? "bad" : "ok");
	return bad || got.size() != pre_lo;
}
"""

RECYCLE = COMMON + r"""
#define KMA_HEAP_RING 1u
#define KMA_CLS_BASE 2u
struct kma_heap { uint32_t flags; uint16_t sb_home[4]; uint32_t sb_state[4], cls[8]; };
static kma_heap h;
static int listed, acts_before;
static void step() { if (acts_before-- == 0) other(); }
static uint32_t ld_relaxed16(const uint16_t *p) { step(); return *p; }
static uint32_t cas_relaxed(uint32_t *p, uint32_t c, uint32_t v)
{
	step();
	uint32_t old = *p;
	if (old == c)
		*p = v;
	return old;
}
static uint32_t *cls_word(kma_heap *, uint32_t, uint32_t shard) { return &h.cls[shard]; }
static void ring_enqueue(kma_heap *, uint32_t, uint32_t) { listed++; }
static void msq_enqueue(kma_heap *, uint32_t) { listed++; }
%s
int main(int, char **argv)
{
	const uint32_t full = st_make(CLS, 7, 7);
	h.flags = atoi(argv[2]);
	h.sb_state[1] = full;
	h.sb_home[1] = 4;
	h.cls[4] = 1 + KMA_CLS_BASE;
	acts_before = atoi(argv[1]); /* accesses before the other thread acts */
	/* the other thread recycles the superblock, unless it is detached; it is
	 * formatted again for the same class, under shard 5, and freed again */
	other = [&] {
		if (h.sb_state[1] != full)
			return;
		h.cls[4] = 0;
		h.sb_home[1] = 5;
		h.cls[5] = 1 + KMA_CLS_BASE;
	};
	sb_recycle(&h, 1, CLS, full);
	bool bad = listed != 1 || h.sb_state[1] != st_make(CLS, 7, 0);
	for (uint32_t w : h.cls)
		bad |= w == 1 + KMA_CLS_BASE; /* no slot names a superblock on the free list */
	printf("%%s\n", bad ? "bad" : "ok");
	return bad;
}
"""


def function(name: str, returns: str = "void") -> str:
    """The text of the function `name` of kma_device.cuh."""
    src = open(DEVICE).read()
    at = src.index(f"__device__ __forceinline__ {returns} {name}(")
    return src[at:src.index("\n}\n", at) + 3]


def build(tmp_path, text: str) -> str:
    cxx = os.environ.get("CXX", "g++")
    if shutil.which(cxx) is None:
        pytest.skip("no C++ compiler")
    (tmp_path / "t.cpp").write_text("#include <cstdlib>\n" + text)
    binary = str(tmp_path / "t")
    subprocess.run([cxx, "-O1", "-std=c++17", "-o", binary, str(tmp_path / "t.cpp")], check=True)
    return binary


def test_a_superblock_is_reserved_from_only_after_its_bitmap(tmp_path):
    """Whoever sees a refilled superblock's state, through its class slot or
    through a hint from an earlier incarnation, sees its bitmap and home."""
    binary = build(tmp_path, FORMAT % function("sb_format"))
    for slots, pre_lo in [(1, 0), (2, 1), (31, 30), (32, 1), (33, 32), (64, 40), (509, 477), (2000, 1)]:
        r = subprocess.run([binary, str(slots), str(pre_lo)], capture_output=True, text=True, timeout=60)
        assert r.returncode == 0, (slots, pre_lo, r.stdout)


@pytest.mark.parametrize("ring", [0, 1])
def test_a_recycled_superblock_leaves_its_current_home(tmp_path, ring):
    """Whenever another thread gets in between: a superblock on the free list
    is in nobody's class slot."""
    binary = build(tmp_path, RECYCLE % (function("sb_detach", "bool") + function("sb_recycle")))
    for before in range(5):
        r = subprocess.run([binary, str(before), str(ring)], capture_output=True, text=True, timeout=60)
        assert r.returncode == 0, (before, r.stdout)
