/* See device_turn.hpp. */

#include "device_turn.hpp"

#include <map>
#include <mutex>

#include "common.hpp"

namespace nemo_b200 {

struct TurnState {
	std::mutex lock;
	std::atomic<int> wanted{0};     /* callers that wait for the turn or for a stay's end */
	cudaEvent_t event = nullptr;    /* the end of the last turn's launches */
	bool pending = false;           /* the event may not have come yet */
	Stay* stay = nullptr;           /* the owner of the last stay */
};

static TurnState&
turnState(int device)
{
	/* never destroyed: simulations may outlive static objects */
	static std::mutex lock;
	static std::map<int, TurnState>& states = *new std::map<int, TurnState>;
	std::lock_guard<std::mutex> guard(lock);
	return states[device];
}

/* The calls below are allowed while another thread captures a stream */
struct RelaxedCapture {
	cudaStreamCaptureMode mode = cudaStreamCaptureModeRelaxed;
	RelaxedCapture() { cudaThreadExchangeStreamCaptureMode(&mode); }
	~RelaxedCapture() { cudaThreadExchangeStreamCaptureMode(&mode); }
};

/* With the turn held: another owner's stay off the device. Counted as wanted
 * meanwhile: the owner's thread, which holds the stay's lock for most of a
 * loop of steps, then gives it up. */
static void
endOther(TurnState& s, const Stay* self)
{
	if(s.stay && s.stay != self) {
		s.wanted++;
		s.stay->endStay();
		s.wanted--;
	}
	s.stay = nullptr;
}

DeviceTurn::DeviceTurn(int device, cudaStream_t stream, const Stay* self) : m_s(turnState(device)), m_stream(stream)
{
	m_s.wanted++;
	m_s.lock.lock();
	m_s.wanted--;
	RelaxedCapture relaxed;
	try {
		endOther(m_s, self);
		if(m_s.event == nullptr) NEMO_CUDA(cudaEventCreateWithFlags(&m_s.event, cudaEventDisableTiming));
		if(m_s.pending) NEMO_CUDA(cudaStreamWaitEvent(m_stream, m_s.event, 0));
	} catch(...) {
		m_s.lock.unlock();
		throw;
	}
}

DeviceTurn::~DeviceTurn()
{
	if(cudaEventRecord(m_s.event, m_stream) == cudaSuccess) m_s.pending = true;
	m_s.lock.unlock();
}

DeviceTurn::TryLock::TryLock(int device, Stay* self) : s(turnState(device)), held(false)
{
	if(s.wanted.load() || !s.lock.try_lock()) return;
	RelaxedCapture relaxed;
	if(s.pending) {
		const cudaError_t e = cudaEventQuery(s.event);
		if(e != cudaSuccess) {
			if(e != cudaErrorNotReady) (void) cudaGetLastError();
			s.lock.unlock();
			return;
		}
		s.pending = false;
	}
	endOther(s, self);
	s.stay = self;
	held = true;
}

DeviceTurn::TryLock::~TryLock()
{
	if(held) s.lock.unlock();
}

const std::atomic<int>*
DeviceTurn::wanted(int device)
{
	return &turnState(device).wanted;
}

void
DeviceTurn::leave(int device, const Stay* self)
{
	TurnState& s = turnState(device);
	std::lock_guard<std::mutex> guard(s.lock);
	if(s.stay == self) s.stay = nullptr;
}

} // namespace nemo_b200
