// A test's view of an engine of the built library: the number of tets that a
// checked build holds indices against.  Lowering it makes the checks reject
// tets whose data is all there.
#include "jgs2_runtime.cpp"

extern "C" unsigned* engine_tet_total(jgs2_batch* batch) { return &batch->b.tetTotal; }
