// Host build of the geometry expansion's counter rule (emit_slot in
// dmsc_b200/csrc/persistent.cuh) for the CPU test.
#include "../../dmsc_b200/csrc/persistent.cuh"

extern "C" int emit_slot_host(int lv, int solo) { return dmsc::emit_slot(lv, solo != 0); }
extern "C" int emit_segs_host() { return dmsc::kEmitSegs; }
